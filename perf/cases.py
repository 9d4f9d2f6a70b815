"""Performance cases of the HDLA operators: what a training or serving program calls, over the sizes it calls them with.

Every case goes through the public entry points (``fused_recurrent_dplr_delta_rule``, ``chunk_hrdplr_delta_rule``,
``chunk_hdla_delta_rule``, ``rms_norm_fused_gate``) with rank 2 and the value distributions of the benchmark
configurations (``hdla_impl_b200/synthetic.py``), drawn on the GPU.

Keys of a case
    path    "decode" / "recurrent"   fused recurrent forward with a carried fp32 state
            "prefill"                chunked forward without gradients, from an initial state to a final state
            "train"                  chunked forward and backward
            "layer"                  the layer's own calls: in-operator a/b parametrisation and l2 norm of k, then
                                     the gated RMS norm over all heads, forward and backward
    B,T,H,K,V    sizes (with seqs > 0: B = 1 and T packed tokens of that many sequences)
    dtype        "bf16" / "fp32" of the tensors;  gk: dtype of the log decay
    gk_div       the log decay is logsigmoid(N(0,1)) / gk_div
    seqs         number of packed sequences, 0 for a uniform batch
    h0           an initial state is given (and, in training, its gradient and the final state's are taken)
    chunk        the chunk size asked for
"""
import math
import random

import torch
import torch.nn.functional as F

from hdla_impl_b200 import chunk_hrdplr_delta_rule, fused_recurrent_dplr_delta_rule
from hdla_impl_b200.layer_ops import chunk_hdla_delta_rule, rms_norm_fused_gate

R = 2                                       # rank of the low-rank term: the HDLA operator's own
_DT = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _case(path, B, T, H, D, dtype="bf16", *, V=None, gk=None, gk_div=16.0, seqs=0, h0=False, chunk=64, name=None):
    c = dict(path=path, B=B, T=T, H=H, K=D, V=D if V is None else V, dtype=dtype, gk=gk or dtype, gk_div=gk_div,
             seqs=seqs, h0=h0, chunk=chunk)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one token for each of a handful of running conversations: what an interactive server does per token and layer
        _case("decode", 4, 1, 16, 128, h0=True, name="decode_b4"),
        # one token for a full serving batch: the decode configuration of the benchmark
        _case("decode", 256, 1, 32, 128, h0=True, name="decode_b256"),
        # short prompts of different lengths through the recurrent path, packed, state carried over
        _case("recurrent", 1, 413, 16, 128, seqs=16, h0=True, name="recurrent_packed"),
        # the prompt of one request, of an odd length
        _case("prefill", 1, 1999, 16, 128, h0=True, name="prefill_b1_t1999"),
        # a server's batch of prompts of different lengths, packed along the time axis
        _case("prefill", 1, 16411, 16, 128, seqs=24, h0=True, name="prefill_packed"),
        # the smallest configuration of the reference: fp32, two short sequences
        _case("train", 2, 256, 4, 64, "fp32", name="train_fp32_small"),
        # fp32 training at the head dims of the large configurations, ragged last chunk
        _case("train", 2, 1000, 8, 128, "fp32", h0=True, name="train_fp32"),
        # the smallest configuration in the training data type: a test run, a toy model
        _case("train", 2, 256, 4, 64, name="train_bf16_small"),
        # heads of 64 channels, odd sequence length, fp32 decay next to bf16 tensors
        _case("train", 4, 2001, 16, 64, gk="fp32", gk_div=4.0, h0=True, name="train_bf16_d64"),
        # the headline training configuration
        _case("train", 8, 4096, 16, 128, name="train_bf16_b8_t4096"),
        # one long document
        _case("train", 1, 65536, 16, 128, name="train_bf16_t65536"),
        # the operator part of one layer of the 2048-wide model, as the layer calls it
        _case("layer", 4, 2048, 16, 128, name="layer_bf16"),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["decode", "recurrent", "prefill", "train", "train", "train32", "layer"])
    H = rng.choice([4, 8, 16, 32])
    D = rng.choice([64, 128, 128])
    h0 = rng.random() < 0.5
    gk_div = rng.choice([4.0, 16.0])
    gk = rng.choice(["bf16", "bf16", "fp32"])
    if path == "decode":
        T = rng.choice([1, 1, 1, 2, 4])
        return _case("decode", _log(rng, 1, 256), T, H, D, rng.choice(["bf16", "bf16", "fp32"]), h0=True, gk_div=gk_div)
    if path == "recurrent":
        if rng.random() < 0.5:
            n = _log(rng, 2, 64)
            return _case("recurrent", 1, n * rng.randint(12, 48) + rng.randint(0, 11), H, D, seqs=n, h0=h0, gk_div=gk_div)
        return _case("recurrent", _log(rng, 1, 32), _log(rng, 9, 128), H, D, rng.choice(["bf16", "fp32"]), h0=h0,
                     gk_div=gk_div)
    if path == "prefill":
        if rng.random() < 0.5:
            n = _log(rng, 2, 32)
            T = n * _log(rng, 64, 1024) + rng.randint(0, 63)
            return _case("prefill", 1, T, H, D, gk=gk, gk_div=gk_div, seqs=n, h0=h0)
        B = _log(rng, 1, 8)
        return _case("prefill", B, _log(rng, 65, min(16384, 2 ** 19 // (B * H))), H, D, gk=gk, gk_div=gk_div, h0=h0)
    if path == "train32":                    # the fp32 pipeline does more per token: smaller totals
        B = _log(rng, 1, 4)
        D = rng.choice([32, 64, 128])
        return _case("train", B, _log(rng, 48, max(64, 2 ** 14 // (B * H))), H, D, "fp32", gk_div=gk_div, h0=h0,
                     chunk=rng.choice([16, 32, 64]))
    if path == "layer":
        B = _log(rng, 1, 8)
        return _case("layer", B, _log(rng, 100, 2 ** 18 // (B * H)), H, D, gk=gk, gk_div=gk_div, h0=h0)
    B = _log(rng, 1, 16)
    D, V = rng.choice([(128, 128), (128, 128), (64, 64), (96, 96), (64, 128)])
    return _case("train", B, _log(rng, 100, min(32768, 2 ** 19 // (B * H))), H, D, V=V, gk=gk, gk_div=gk_div, h0=h0)


def _offsets(case):
    """Offsets of a packed batch: lengths around the mean, from a quarter of it to about twice it.  They belong to the
    case, not to the inputs."""
    n, T = case["seqs"], case["T"]
    rng = random.Random(1000 * n + T)
    w = [rng.uniform(0.25, 1.75) for _ in range(n)]
    cut, total, acc = [0], sum(w), 0.0
    for x in w[:-1]:
        acc += x
        cut.append(max(cut[-1] + 1, int(T * acc / total)))
    return cut + [T]


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    B, T, H, K, V = (case[n] for n in ("B", "T", "H", "K", "V"))
    dt, gdt = _DT[case["dtype"]], _DT[case["gk"]]
    path = case["path"]

    def rn(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    s = dict(case=case, path=path, chunk=case["chunk"])
    s["q"] = F.normalize(rn(B, T, H, K), dim=-1).to(dt)
    s["v"] = rn(B, T, H, V).to(dt)
    s["gk"] = (F.logsigmoid(rn(B, T, H, K)) / case["gk_div"]).to(gdt)
    if path == "layer":
        s["k"] = F.silu(rn(B, T, H, K)).to(dt)                     # un-normalised: the operator normalises it
        s["beta"] = (2 * torch.sigmoid(rn(B, T, H, 1))).to(dt)
        s["gate"] = rn(B, T, H * V).to(dt)
        s["weight"] = (1 + 0.02 * rn(H * V)).to(dt)
        s["do"] = rn(B, T, H * V).to(dt)
    else:
        s["k"] = F.normalize(rn(B, T, H, K), dim=-1).to(dt)
        s["a"] = (-F.normalize(rn(B, T, R, H, K), dim=-1)).reshape(B, T * R, H, K).to(dt)
        b = F.normalize(rn(B, T, R, H, K), dim=-1) * torch.sigmoid(rn(B, T, R, H, 1))
        s["b"] = b.reshape(B, T * R, H, K).to(dt)
        s["do"] = rn(B, T, H, V).to(dt) if path == "train" else None
    s["cu"] = None
    n_states = B
    if case["seqs"]:
        offs = _offsets(case)
        n_states = case["seqs"]
        s["cu"] = torch.tensor(offs, dtype=torch.int64, device=dev) if path == "recurrent" else offs
    s["h0"] = s["dht"] = None
    if case["h0"]:
        s["h0"] = rn(n_states, H, K, V) * 0.02
        s["dht"] = rn(n_states, H, K, V) * 0.1
    if path in ("train", "layer"):
        names = ["q", "k", "v", "a", "b", "gk"] if path == "train" else ["q", "k", "v", "beta", "gk", "gate", "weight"]
        s["leaves"] = [s[n].requires_grad_(True) for n in names]
        if case["h0"]:
            s["leaves"].append(s["h0"].requires_grad_(True))
    return s


def run(s):
    path, h0 = s["path"], s["h0"]
    if path in ("decode", "recurrent"):
        return fused_recurrent_dplr_delta_rule(s["q"], s["k"], s["v"], s["a"], s["b"], s["gk"], R, initial_state=h0,
                                               output_final_state=True, cu_seqlens=s["cu"])
    if path == "prefill":
        with torch.no_grad():
            return chunk_hrdplr_delta_rule(s["q"], s["k"], s["v"], s["a"], s["b"], s["gk"], R, initial_state=h0,
                                           output_final_state=True, chunk_size=s["chunk"], cu_seqlens=s["cu"])
    if path == "train":
        o, ht = chunk_hrdplr_delta_rule(s["q"], s["k"], s["v"], s["a"], s["b"], s["gk"], R, initial_state=h0,
                                        output_final_state=True, chunk_size=s["chunk"])
        y = o
    else:
        o, ht = chunk_hdla_delta_rule(s["q"], s["k"], s["v"], s["beta"], s["gk"], scale=1.0, initial_state=h0,
                                      output_final_state=True, normalize_k=True)
        y = rms_norm_fused_gate(o.flatten(2), s["gate"], s["weight"])
    if h0 is None:
        grads = torch.autograd.grad(y, s["leaves"], s["do"])
    else:
        grads = torch.autograd.grad([y, ht], s["leaves"], [s["do"], s["dht"]])
    return y.detach(), ht.detach(), grads


def work(case):
    """Bytes: every input once, every output (with its gradients) once.  Operations: the recurrence itself, which per
    token and head applies two rank-one updates, the decay and the new key-value pair to a K x V state and reads it
    once; backward twice that."""
    B, T, H, K, V = (case[n] for n in ("B", "T", "H", "K", "V"))
    es, gs = (2 if case["dtype"] == "bf16" else 4), (2 if case["gk"] == "bf16" else 4)
    n = B * T * H
    states = (case["seqs"] or B) * H * K * V * 4
    step = (4 * R + 5) * K * V
    path = case["path"]
    tensors = (2 + (2 * R if path != "layer" else 0)) * K * es + V * es + K * gs + (es if path == "layer" else 0)
    out = V * es
    state_io = states * (2 if case["h0"] else 1)
    if path in ("decode", "recurrent", "prefill"):
        return {"bytes": n * (tensors + out) + state_io, "flops": n * step}
    moved = n * (2 * tensors + 2 * out) + state_io * (2 if case["h0"] else 1)
    if path == "layer":
        moved += n * 2 * V * es                      # the gate and its gradient
    return {"bytes": moved, "flops": 3 * n * step}


def tolerance(case):
    """fp32: rounding of sums of a few hundred products, carried through the chunks.  bf16: the recurrent path computes in
    fp32 and rounds its output once; the chunked path's operands between the products are bf16 too, which puts its
    outputs 2e-3 to 6e-3 from the exact ones (the layer's beta gradient, a difference of large sums, 1.2e-2)."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["path"] in ("decode", "recurrent"):
        return {"rel": 2e-3, "max": 1e-2}
    return {"rel": 2e-2 if case["path"] == "layer" else 1e-2, "max": 0.3}
