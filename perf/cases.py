"""Workloads of the slot-memory operators, as a program that uses the package runs them.

Each case is one call (or one replay, or one forward and backward pass) through the public entry points:
``random_access_memory_attention``, ``topk_addr`` and ``DecodeGraph``.  Sizes are those of the package's own
configurations, tests and benchmark, and sizes between them:

  kind      decode   one token per sequence on a kept state (T = 1, in place)
            graph    sixteen decode steps replayed from a CUDA graph, with the head norm and the output gate
            prefill  a prompt, on a zero state or continuing a kept one
            train    forward and backward
            address  Top-K address decoding alone
  family    (U digits, radix P, K addresses): see FAMILIES
  B T H C   batch, tokens, heads, channels of a value row
  dtype     of logits, values and forget gates; the state is always float32
  pad       left-padded batch: a token mask with the matching positions
  carry     prefill continues a kept state in place; train starts from a given state and also differentiates
            with respect to it
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("ram-net_b200"))

import ramnet_ops  # noqa: E402
from ramnet_ops.decode_graph import DecodeGraph  # noqa: E402

# (U, P, K) -> slots per head: 256, 512, 1024, 4096 (five ways), and for addressing alone 32768 (two ways)
FAMILIES = ((2, 16, 4), (3, 8, 8), (2, 32, 8), (2, 64, 8), (2, 64, 16), (2, 64, 32), (4, 8, 16))
ADDRESS_ONLY = ((3, 32, 8), (5, 8, 8))
GRAPH_STEPS = 16
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _case(kind, B, T, H, family, C, dtype, pad=False, carry=False, mass_aware=False, re_norm=0.0, **more):
    U, P, K = family
    return dict(more, kind=kind, B=B, T=T, H=H, U=U, P=P, K=K, C=C, dtype=dtype, pad=pad, carry=carry,
                mass_aware=mass_aware, re_norm=re_norm)


def listed():
    return [
        # one user's generation loop, one layer, called token by token: nothing but latency
        _case("decode", 1, 1, 16, (2, 64, 16), 128, "bf16", carry=True, name="decode_one"),
        # a serving batch at the largest state (8.6 GB per layer), called token by token
        _case("decode", 256, 1, 16, (2, 64, 16), 128, "bf16", carry=True, name="decode_batch"),
        # radix-8 addresses with the default K, mass-aware reads, a batch in which some sequences have ended
        _case("decode", 48, 1, 8, (3, 8, 8), 64, "f16", pad=True, carry=True, mass_aware=True, re_norm=0.5,
              name="decode_radix8"),
        # the generation loop of one layer of the full model at batch 64, replayed from a graph
        _case("graph", 64, 1, 16, (2, 64, 16), 128, "bf16", carry=True, name="decode_graph"),
        # the single-layer float32 configuration
        _case("prefill", 1, 512, 4, (2, 16, 4), 64, "f32", name="prefill_small"),
        # one prompt, or the next part of one, on a kept state
        _case("prefill", 1, 1999, 16, (2, 64, 16), 128, "bf16", carry=True, name="prefill_prompt"),
        # a left-padded batch of prompts with the default K and mass-aware reads
        _case("prefill", 6, 777, 16, (2, 64, 8), 128, "f16", pad=True, mass_aware=True, name="prefill_padded"),
        # the long-context batch of the benchmark
        _case("prefill", 8, 16384, 16, (2, 64, 16), 128, "bf16", name="prefill_long"),
        # float32 training at the single-layer size, carried state (truncated back-propagation through time)
        _case("train", 2, 500, 4, (2, 16, 4), 64, "f32", pad=True, carry=True, name="train_small"),
        # one layer of the full model, training batch
        _case("train", 8, 2048, 16, (2, 64, 16), 128, "bf16", name="train_layer"),
        # the long-context batch, forward and backward
        _case("train", 8, 16384, 16, (2, 64, 16), 128, "bf16", name="train_long"),
        # addressing alone, 32768 slots per head
        _case("address", 8, 8192, 16, (3, 32, 8), 0, "bf16", name="address"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("decode", "graph", "prefill", "prefill", "train", "train", "address"))
    family = rng.choice(FAMILIES + (ADDRESS_ONLY if kind == "address" else ()))
    U, P, K = family
    H = rng.choice((4, 8, 16))
    C = 0 if kind == "address" else rng.choice((64, 128, 128, 256))
    dtype = rng.choice(("bf16", "bf16", "f16", "f32"))
    pad = kind in ("decode", "prefill", "train") and rng.random() < 0.3
    carry = kind in ("decode", "graph") or (kind != "address" and rng.random() < 0.5)
    mass_aware = kind != "address" and rng.random() < 0.2
    re_norm = rng.choice((0.0, 0.0, 0.5, 1.0))
    if kind in ("decode", "graph"):
        # no state above that of the largest listed case
        B, T = _log_int(rng, 1, min(256, 256 * 16 * 4096 * 128 // (H * P ** U * C))), 1
    else:
        # tokens x heads x channels x K stay below an eighth of the largest listed case
        most = 8 * 16384 * 16 * 128 * 16 // (8 * H * max(C, 32) * K)
        T = _log_int(rng, 32, min(16384, most))
        B = _log_int(rng, 1, max(1, min(16, most // T)))
    return _case(kind, B, T, H, family, C, dtype, pad=pad, carry=carry, mass_aware=mass_aware, re_norm=re_norm)


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    dt = DTYPES[c["dtype"]]
    B, T, H, U, P, K, C = (c[k] for k in "BTHUPKC")
    A = P ** U

    def normal(*shape, std=1.0, dtype=dt):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.float32).mul_(std).to(dtype)

    s = {"case": c}
    if c["kind"] == "address":
        # logits as the projection leaves them, (B,T,H,U,P); the entry point takes the time axis last
        s["addr"] = normal(B, T, H, U, P, std=1.5).permute(0, 2, 3, 4, 1)
        s["pos"] = torch.arange(T, device=dev).view(1, T).expand(B, T).contiguous()
        return s

    lead = (GRAPH_STEPS, B) if c["kind"] == "graph" else (B, T)
    s["w"], s["r"] = normal(*lead, H, U, P), normal(*lead, H, U, P)
    s["x"] = normal(*lead, H, C)
    s["gamma"] = torch.sigmoid(normal(*lead, H, dtype=torch.float32) + 1.0).to(dt)
    s["mask"] = s["pos"] = s["state"] = None
    if c["carry"]:
        # a state that has been written to: rows of some tenths, masses from almost empty to full
        s["state"] = (normal(B, H, A, C, std=0.1, dtype=torch.float32),
                      torch.rand(B, H, A, generator=g, device=dev).add_(0.01))
    if c["kind"] == "decode":
        s["pos"] = torch.randint(0, 4 * A, (B, 1), generator=g, device=dev)
        if c["pad"]:  # sequences that have ended: an eighth of the batch
            s["mask"] = torch.rand(B, 1, generator=g, device=dev) >= 0.125
    elif c["kind"] == "graph":
        pos = torch.randint(0, 4 * A, (B,), generator=g, device=dev, dtype=torch.int32)
        s["graph"] = DecodeGraph(s["w"], s["r"], s["x"], s["gamma"], s["state"][0], s["state"][1], pos, embed_num=H // 2,
                                 top_k=K, w_re_norm=c["re_norm"], r_re_norm=c["re_norm"], mass_aware=c["mass_aware"],
                                 norm_weight=normal(C, std=0.1, dtype=torch.float32) + 1.0,
                                 gate_logits=normal(GRAPH_STEPS, B, H, C))
    elif c["pad"]:
        length = torch.randint(max(1, T // 2), T + 1, (B, 1), generator=g, device=dev)
        s["mask"] = torch.arange(T, device=dev).view(1, T) >= T - length
        s["pos"] = (s["mask"].long().cumsum(-1) - 1).clamp_(min=0)
    if c["kind"] == "train":
        s["d_y"] = normal(B, T, H, C)
        s["leaves"] = [t.requires_grad_(True) for t in (s["w"], s["r"], s["x"], s["gamma"])]
        s["up"] = [s["d_y"]]
        if c["carry"]:
            s["leaves"] += [t.requires_grad_(True) for t in s["state"]]
            s["up"] += [normal(B, H, A, C, std=0.1, dtype=torch.float32), normal(B, H, A, std=0.1, dtype=torch.float32)]
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "address":
        return ramnet_ops.topk_addr(s["addr"], c["H"] // 2, s["pos"], c["K"], c["re_norm"])
    if c["kind"] == "graph":
        return {"y": s["graph"].replay(), "slot": s["graph"].slot, "mass": s["graph"].mass}
    inplace = c["kind"] == "decode" or (c["kind"] == "prefill" and c["carry"])
    y, state = ramnet_ops.random_access_memory_attention(
        s["w"], s["r"], s["x"], s["gamma"], s["state"], mask=s["mask"], embed_num=c["H"] // 2, position_ids=s["pos"],
        top_k=c["K"], top_k_re_norm=c["re_norm"], mass_aware=c["mass_aware"], inplace=inplace)
    if c["kind"] != "train":
        return y, state
    outputs = (y, *state) if c["carry"] else (y,)
    return y.detach(), [t.detach() for t in state], torch.autograd.grad(outputs, s["leaves"], s["up"])


def work(case):
    c = case
    B, T, H, U, P, K, C = (c[k] for k in "BTHUPKC")
    A, size = P ** U, 4 if c["dtype"] == "f32" else 2
    n = B * T * H * (GRAPH_STEPS if c["kind"] == "graph" else 1)  # token-heads
    softmax = 4 * U * P  # maximum, difference, exponential and sum of a logit
    if c["kind"] == "address":
        return {"bytes": n * U * P * size + B * T * 8 + n * K * 8, "flops": n * softmax}
    logits, row = 2 * n * U * P * size, n * C * size
    inputs = logits + row + n * size + (B * T * 9 if c["pad"] else 0)
    update = n * C * K * 5  # a write: difference, product, sum; a read: product, sum
    if c["kind"] in ("decode", "graph"):
        # K rows read and written, K rows read, with their masses
        state = n * K * (3 * C + 2) * 4
        return {"bytes": inputs + row + state + (row if c["kind"] == "graph" else 0), "flops": update + 2 * n * softmax}
    # in place, the rows that are touched; else the whole state: written, and read unless it starts from zero
    whole = B * H * A * (C + 1) * 4
    touched = B * H * min(A, T * K) * (C + 1) * 4
    if c["kind"] == "prefill":
        return {"bytes": inputs + row + (2 * touched if c["carry"] else whole), "flops": update + 2 * n * softmax}
    # forward and backward: d_y in, gradients of logits, values and gates out; with a carried state also its gradients
    state = 4 * whole if c["carry"] else whole
    return {"bytes": inputs + row + row + logits + row + n * size + state, "flops": 3 * update + 6 * n * softmax}


def tolerance(case):
    if case["kind"] == "address":
        return {"rel": 1e-5}  # indices are the same; weights are float32 whatever the logits are
    if case["dtype"] != "f32":
        # results are rounded to the type of the values (and gradients to that of what they belong to)
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
    # 32-bit sums; the gradients of a softmax and of the forgetting factor are differences of such sums
    return {"rel": 1e-4 if case["kind"] == "train" else 1e-5}
