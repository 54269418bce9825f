"""The calls a program makes of this framework, at the sizes it makes them.

A case is one training step (forward and gradients), one evaluation (forward alone) or one
host-buffer step of the pair-biased attention of AlphaFold-3-like models:

    B, S, N, H, D   batch, rows of the MSA / of the pair representation, residues, heads, head dim
    mode            "train": forward + gradients of q, k, v, pair bias (and gate)
                    "infer": forward without gradients
                    "host":  forward + gradients for tensors that live in host memory
    view            where q, k, v lie: "plain" contiguous [B, S, N, H, D]; "ending" stored
                    [B, N, S, H, D] (triangle attention around the ending node); "fused" sliced out
                    of one projection's output [B, S, N, 3, H, D]
    gate            sigmoid gate fused into the call
    bias            dtype in which pair bias and residue mask are handed over, "bf16" or "fp32"
    mask            "valid", "tail" (padded crop) or "random" (a share of the residues missing)

Ranges: D in 16, 32, 64, 96, 128; N from 40 to 1024 in steps of 8, tile multiples or ragged; S from 1
to 1024; H from 1 to 16; B from 1 to 8, up to the work of the largest listed case.
"""
import os
import sys

import torch

# the package's modules are imported from its folder; the repository's root is the working folder
sys.path.insert(0, os.path.abspath("megakernel-exploration_b200"))

from tk_evo_attention_layer import EvoAttention, HostStreamedEvoAttention, TKEvoAttention  # noqa: E402

DEV = "cuda"


def _case(name, mode, B, S, N, H, D, view="plain", gate=False, bias="bf16", mask="tail"):
    c = {"mode": mode, "B": B, "S": S, "N": N, "H": H, "D": D, "view": view, "gate": gate, "bias": bias, "mask": mask}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small crop while debugging or fine-tuning: latency, launches and host work are all of it
        _case("small_crop_train", "train", 1, 32, 64, 4, 32, mask="random"),
        # single-row pair-biased attention at the short end of the sequence-length sweep
        _case("single_row_n128_train", "train", 4, 1, 128, 16, 64, mask="random"),
        # ... and at its long end
        _case("single_row_n1024_train", "train", 4, 1, 1024, 16, 64, mask="random"),
        # evaluation of a mid-sized single-row stack; the pair bias is handed over in bf16
        _case("single_row_n512_infer", "infer", 4, 1, 512, 16, 64, mask="random"),
        # MSA row attention, the benchmark's training step: a padded crop of 384 residues
        _case("msa_row_train", "train", 1, 512, 384, 8, 32),
        # the same block in evaluation
        _case("msa_row_infer", "infer", 1, 512, 384, 8, 32),
        # triangle attention around the ending node with its gate, mask and bias kept in fp32
        _case("triangle_ending_gated_train", "train", 1, 384, 384, 4, 32, view="ending", gate=True, bias="fp32"),
        # triangle attention of an uncropped, ragged chain; q, k, v sliced out of one projection
        _case("triangle_ragged_fused_train", "train", 1, 200, 200, 4, 32, view="fused", mask="valid"),
        # a large MSA at 768 residues
        _case("large_msa_train", "train", 1, 1024, 768, 8, 32),
        # triangle attention of a long chain at head dim 64: the largest step
        _case("long_triangle_train", "train", 1, 1024, 1024, 4, 64, mask="random"),
        # wide heads
        _case("wide_heads_train", "train", 1, 128, 768, 4, 128),
        # a caller whose tensors live in host memory, copied in and out while the kernels run
        _case("host_buffers", "host", 1, 128, 384, 8, 32),
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    mode = rng.choices(("train", "infer", "host"), (60, 30, 10))[0]
    D = rng.choices((16, 32, 64, 96, 128), (10, 45, 25, 8, 12))[0]
    N = 8 * max(1, round(_log_uniform(rng, 40, 1024) / 8))
    H = rng.choice((1, 2, 3, 4, 4, 6, 8, 8, 12, 16))
    if rng.random() < 0.3:
        B, S = rng.choice((1, 2, 3, 4, 6, 8)), 1
    else:
        B, S = rng.choice((1, 1, 1, 2)), max(2, round(_log_uniform(rng, 2, 1024)))
    view, gate, bias = "plain", False, rng.choice(("bf16", "bf16", "fp32"))
    if mode == "host":
        bias = "bf16"
    else:
        view = rng.choices(("plain", "ending", "fused"), (60, 20, 20))[0] if S > 1 else rng.choice(("plain", "plain", "fused"))
        gate = rng.random() < 0.25
    padded = 128 * -(-N // 128)
    most_logits, most_values = 2 ** 31, (2 ** 24 if mode == "host" else 2 ** 28)
    while B * S * H * padded * padded > most_logits or B * S * N * H * D > most_values:
        if S > 2:
            S = max(2, int(S * 0.7))
        else:
            H = max(1, H - 1)
    return _case(None, mode, B, S, N, H, D, view, gate, bias, rng.choice(("valid", "tail", "random")))


def _mask(case, gen):
    B, S, N = case["B"], case["S"], case["N"]
    keep = torch.ones((B, S, N), dtype=torch.bool, device=DEV)
    if case["mask"] == "tail":
        # crops of one batch share their padding; a chain is at least seven eighths of its crop
        length = N - (torch.rand((B, 1, 1), generator=gen, device=DEV) * (N / 8)).long()
        keep = (torch.arange(N, device=DEV) < length).expand(B, S, N).clone()
    elif case["mask"] == "random":
        keep = torch.rand((B, S, N), generator=gen, device=DEV) < 0.9
    keep[..., 0] = True
    return torch.where(keep, 0.0, -1e9).reshape(B, S, 1, 1, N)


def prepare(case, seed):
    B, S, N, H, D = (case[k] for k in "BSNHD")
    gen = torch.Generator(device=DEV).manual_seed(seed)
    bf = torch.bfloat16

    def normal(*shape, std=1.0, dtype=bf):
        return (torch.randn(shape, generator=gen, device=DEV) * std).to(dtype)

    pair = torch.float32 if case["bias"] == "fp32" else bf
    if case["view"] == "fused":
        q, k, v = normal(B, S, N, 3, H, D, std=0.5).unbind(3)
    elif case["view"] == "ending":
        q, k, v = (normal(B, N, S, H, D, std=0.5).transpose(1, 2) for _ in range(3))
    else:
        q, k, v = (normal(B, S, N, H, D, std=0.5) for _ in range(3))
    mask = _mask(case, gen).to(pair)
    bias = normal(B, 1, H, N, N, dtype=pair)

    if case["mode"] == "host":
        d_o = normal(B, S, N, H, D)
        host = [t.cpu().pin_memory() for t in (q, k, v, mask, bias, d_o)]
        out = {n: torch.empty((B, S, N, H, D), dtype=bf).pin_memory() for n in ("o", "dq", "dk", "dv")}
        out["dbias"] = torch.empty((B, 1, H, N, N), dtype=torch.float32).pin_memory()
        return {"mode": "host", "host": host, "out": out, "engine": HostStreamedEvoAttention(DEV, chunk_rows=64)}

    state = {"mode": case["mode"], "q": q, "k": k, "v": v, "mask": mask, "bias": bias, "gate": None}
    if case["gate"]:
        gate = normal(B, N, S, H, D).transpose(1, 2) if case["view"] == "ending" else normal(B, S, N, H, D)
        state["gate"] = gate
        state["module"] = EvoAttention()
    if case["mode"] == "train":
        d_o = normal(B, N, S, H, D).transpose(1, 2) if case["view"] == "ending" else normal(B, S, N, H, D)
        state["d_o"] = d_o
        for n in ("q", "k", "v", "bias", "gate"):
            if state[n] is not None:
                state[n] = state[n].detach().requires_grad_(True)
    return state


def _attention(s):
    if s["gate"] is not None:
        return s["module"](s["q"], s["k"], s["v"], s["mask"], s["bias"], gate=s["gate"])
    return TKEvoAttention.apply(s["q"], s["k"], s["v"], s["mask"], s["bias"])


def run(state):
    if state["mode"] == "host":
        state["engine"].run(*state["host"], state["out"])
        return state["out"]
    if state["mode"] == "infer":
        with torch.no_grad():
            return _attention(state)
    o = _attention(state)
    wrt = [state[n] for n in ("q", "k", "v", "bias", "gate") if state[n] is not None]
    return (o.detach(),) + torch.autograd.grad(o, wrt, state["d_o"])


def work(case):
    """Bytes: q, k, v, mask, pair bias (and gate, dO) read once, O (and every gradient) written once.
    FLOPs: 4 B S H N^2 D for the forward, 10 for the backward."""
    B, S, N, H, D = (case[k] for k in "BSNHD")
    acts, pair = 2 * B * S * N * H * D, B * H * N * N
    each = 4 if case["bias"] == "fp32" else 2
    flops = 4.0 * B * S * H * N * N * D
    moved = (5 if case["gate"] else 4) * acts + each * (B * S * N + pair)
    if case["mode"] != "infer":
        flops *= 3.5
        moved += (5 if case["gate"] else 4) * acts + (4 if case["mode"] == "host" else each) * pair
    return {"bytes": float(moved), "flops": flops}


def tolerance(case):
    # bf16 products of probabilities and gradients, bf16 outputs; the largest single difference is a few
    # bf16 steps of that value or of the result's root mean square
    return {"rel": 1e-2, "max": 0.1}
