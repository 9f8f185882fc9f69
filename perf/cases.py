"""What a user of this library has it do, as a set of measurable cases.

Three ways in, all through the public module ``flash_tt_attn``:

  infer   one forward call under ``torch.no_grad()``
  train   one forward call and the gradients of q, k, v and the pair bias
  stream  ``attention_fwd_bwd_streamed``: forward and backward of tensors in pinned host memory

A case says which of them, the sizes (B, H, L1, L2, D), the 16-bit type, how keys are masked
(``none``; ``key``: the boolean ``key_mask`` argument; ``bias``: -1e9 added to the bias columns of the
masked keys, the way pair-stack code writes it) and whether q, k, v are the ending-node views
(stored with L1 and L2 exchanged and handed over through ``transpose(2, 3)``, as is dO).
Values are N(0, 1), or ``std`` / ``bias_std`` where a case says so; a mask drops 10 % of the keys.
"""
import math

import torch

import flash_tt_attn

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
MASK_FRACTION = 0.1


def _case(name, mode, B, H, L1, L2, D, dtype, mask="none", ending=False, std=1.0, bias_std=1.0):
    return {"name": name, "mode": mode, "B": B, "H": H, "L1": L1, "L2": L2, "D": D, "dtype": dtype,
            "mask": mask, "ending": ending, "std": std, "bias_std": bias_std}


def listed():
    return [
        # a short chain, scored once: nothing but launches and host time
        _case("infer_l64", "infer", 1, 4, 64, 64, 32, "fp16"),
        # the same chain in a training step (unit tests and tiny crops of a fine-tuning run)
        _case("train_l64", "train", 1, 4, 64, 64, 32, "bf16"),
        # the README's benchmark shape
        _case("train_readme_l256", "train", 4, 8, 256, 256, 32, "fp16"),
        # the same with the wider head
        _case("train_d64_l256", "train", 4, 8, 256, 256, 64, "bf16"),
        # a padded batch of two chains: ragged length, boolean key mask
        _case("train_ragged_l200", "train", 2, 4, 200, 200, 32, "bf16", mask="key"),
        # inference on a chain of odd length with unresolved residues masked out
        _case("infer_odd_l317", "infer", 1, 8, 317, 317, 32, "fp16", mask="key"),
        # a training crop, masked residues written into the bias
        _case("train_crop_l384", "train", 1, 4, 384, 384, 32, "bf16", mask="bias"),
        # the ending-node half of a pair-stack block: strided views in, strided gradients out
        _case("train_ending_l512", "train", 1, 4, 512, 512, 32, "bf16", ending=True),
        # the headline training shape
        _case("train_l768", "train", 1, 4, 768, 768, 32, "bf16"),
        # inference on a large complex: normalised q, k, v, a wide bias
        _case("infer_l1024", "infer", 1, 4, 1024, 1024, 32, "bf16", std=1.0 / math.sqrt(32.0), bias_std=2.0),
        # the headline shape with tensors that live in host memory
        _case("stream_l768", "stream", 1, 4, 768, 768, 32, "bf16"),
        # long-sequence training, the largest configuration
        _case("train_l2048_d64", "train", 1, 8, 2048, 2048, 64, "bf16"),
    ]


# a drawn case costs at most what the largest listed one does, in arithmetic and in memory
_MOST_SCORES = 8 * 2048 ** 3 * 64
_MOST_ELEMS = 8 * 2048 ** 2 * 64
_MOST_STREAMED = 4 * 768 ** 2 * 32


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        mode = rng.choice(["train"] * 6 + ["infer"] * 4 + ["stream"])
        L2 = _log_int(rng, 16, 2048)
        kind = rng.random()
        if kind < 0.4:  # crops come in whole blocks
            L2 = max(16, L2 // 64 * 64) if L2 >= 64 else max(16, L2 // 16 * 16)
        elif kind < 0.7 or mode == "stream":  # padded to the vector width
            L2 = (L2 + 7) // 8 * 8
        # the square pair representation, one GPU's share of its rows, or any number of rows
        shape = rng.random()
        if shape < 0.6:
            L1 = L2
        elif shape < 0.85:
            L1 = max(1, L2 // rng.choice([2, 4, 8]))
        else:
            L1 = _log_int(rng, 1, 1024)
        B, H = rng.choice([1, 1, 1, 2, 4]), rng.choice([1, 2, 4, 4, 8, 8, 16])
        D = rng.choice([32, 32, 32, 64])
        dtype = rng.choice(["bf16", "bf16", "fp16"])
        mask = "none" if mode == "stream" else rng.choice(["none", "none", "key", "bias"])
        ending = mode != "stream" and rng.random() < 0.25
        elems = B * H * L1 * L2 * D
        if elems * L2 > _MOST_SCORES or elems > (_MOST_STREAMED if mode == "stream" else _MOST_ELEMS):
            continue
        c = _case("", mode, B, H, L1, L2, D, dtype, mask=mask, ending=ending)
        del c["name"]
        return c


def prepare(case, seed):
    B, H, L1, L2, D = (case[k] for k in ("B", "H", "L1", "L2", "D"))
    dtype = _DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, std=1.0):
        x = torch.randn(shape, device="cuda", dtype=dtype, generator=g)
        return x if std == 1.0 else x.mul_(std)

    rows = (L2, L1) if case["ending"] else (L1, L2)
    t = {n: randn(B, H, *rows, D, std=case["std"]) for n in ("q", "k", "v")}
    t["bias"] = randn(B, H, L2, L2, std=case["bias_std"])
    if case["mode"] != "infer":
        t["do"] = randn(B, H, *rows, D)
    state = {"mode": case["mode"], "ending": case["ending"], "scale": D ** -0.5, "key_mask": None}
    if case["mask"] != "none":
        keep = torch.rand(B, L2, device="cuda", generator=g) >= MASK_FRACTION
        keep[:, 0] = True  # never a row without a key
        if case["mask"] == "key":
            state["key_mask"] = keep
        else:
            t["bias"].add_(torch.where(keep, 0.0, -1.0e9)[:, None, None, :].to(dtype))
    if case["mode"] == "stream":
        state["host"] = {n: x.cpu().pin_memory() for n, x in t.items()}
        state["out"] = {n: torch.empty((B, H, L1, L2, D), dtype=dtype).pin_memory() for n in ("o", "dq", "dk", "dv")}
        state["out"]["dbias"] = torch.empty((B, H, L2, L2), dtype=dtype).pin_memory()
        return state
    if case["mode"] == "train":
        for n in ("q", "k", "v", "bias"):
            t[n].requires_grad_()
    state.update(t)
    return state


def run(state):
    if state["mode"] == "stream":
        flash_tt_attn.attention_fwd_bwd_streamed(state["host"], state["scale"], state["out"])
        return state["out"]
    with torch.set_grad_enabled(state["mode"] == "train"):
        qkv = [state[n] for n in ("q", "k", "v")]
        if state["ending"]:
            qkv = [x.transpose(2, 3) for x in qkv]
        o = flash_tt_attn.attention(*qkv, state["bias"], state["scale"], key_mask=state["key_mask"])
        if state["ending"]:
            o = o.transpose(2, 3)
    if state["mode"] == "infer":
        return o
    dq, dk, dv, dbias = torch.autograd.grad(o, [state[n] for n in ("q", "k", "v", "bias")], state["do"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv, "dbias": dbias}


def work(case):
    """q, k, v and the bias in and O out; a training step also takes dO and gives the four gradients.
    Two matrix products per score forward, five more backward."""
    B, H, L1, L2, D = (case[k] for k in ("B", "H", "L1", "L2", "D"))
    rows, plane = B * H * L1 * L2 * D, B * H * L2 * L2
    fwd = 4.0 * rows * L2
    if case["mode"] == "infer":
        return {"bytes": 2 * (4 * rows + plane), "flops": fwd}
    return {"bytes": 2 * (8 * rows + 2 * plane), "flops": 3.5 * fwd}


def tolerance(case):
    """Probabilities, outputs and gradients are rounded to 8 (bf16) or 11 (fp16) bits; single values of
    peaked rows stray further, relative to the root mean square, than the whole does."""
    return {"rel": 1e-2, "max": 0.6} if case["dtype"] == "bf16" else {"rel": 2e-3, "max": 0.15}
