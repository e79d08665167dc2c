"""The work whose speed is watched: decoding, batched decoding and prompts of every model family.

A case is a dict of plain values; ``prepare`` builds the model (random weights of a real shape), the
state of the sequences and the generator that a serving program keeps, ``run`` makes one call of
that generator, ``exact`` computes the same in 64 bits with plain torch.

Kinds of cases:

* ``decode``: one token of one sequence that already holds ``position`` tokens (llama and layer-list
  models), launched eagerly or replayed as a CUDA graph;
* ``batch``: one token of each of ``sequences`` independent sequences of ragged lengths (llama);
* ``prompt``: ``tokens`` tokens at once after ``position`` earlier ones.

Weights are normal, with the matrices that write the residual stream scaled down by the depth (the
usual initialisation of deep decoders); norms and scales lie around their neutral values.  Cached
keys and values of llama cases are N(0, 1); layer-list cases feed a prompt for them.
"""

from __future__ import annotations

import math
import zlib

import torch

from megakernels_b200.demos.latency.scheduler import LatencyScheduleOptions, pick_num_attention_partitions
from megakernels_b200.dispatch import make_generator
from megakernels_b200.dumalix import DumalixForCausalLM
from megakernels_b200.llama import LlamaConfig, LlamaForCausalLM, StackedParams
from megakernels_b200.model_types import ExtraModelConfig
from megakernels_b200.torirax import ToriraxForCausalLM

VOCAB = 128256
LLAMA = {
    "llama-1b": dict(width=2048, ff=8192, layers=16, heads=32, kv_heads=8, dim=64, tied=True, factor=32.0),
    "llama-8b": dict(width=4096, ff=14336, layers=32, heads=32, kv_heads=8, dim=128, tied=False, factor=8.0),
}
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


# ---- cases --------------------------------------------------------------------------------- #
def listed() -> list[dict]:
    return [
        # a chat's first answer: the smallest step, where launches and hand-overs count
        dict(name="llama-1b-chat", kind="decode", model="llama-1b", layers=16, position=47, graph=True),
        # the headline benchmark: 8B widths at full depth, about a thousand cached positions
        dict(name="llama-8b-decode", kind="decode", model="llama-8b", layers=32, position=1029, graph=False),
        # a long document: the cache outweighs the weights
        dict(name="llama-1b-long", kind="decode", model="llama-1b", layers=16, position=65001, graph=True),
        # a few users at once; depth cut (a layer is what repeats)
        dict(name="llama-8b-batch-7", kind="batch", model="llama-8b", layers=8, sequences=7, longest=4096),
        # a server's full batch
        dict(name="llama-8b-batch-64", kind="batch", model="llama-8b", layers=6, sequences=64, longest=4096),
        # a prompt before the first answer
        dict(name="llama-1b-prompt", kind="prompt", model="llama-1b", layers=16, position=0, tokens=501),
        # recurrent layers and windowed differential attention: one token past the window
        dict(name="torirax-1b-decode", kind="decode", model="torirax-1b", dtype="bf16", position=4096, graph=True),
        # the same in float32 (the exact build), a prompt of ordinary length
        dict(name="torirax-1b-f32-prompt", kind="prompt", model="torirax-1b", dtype="f32", position=0, tokens=300),
        # a full portion through the large widths
        dict(name="torirax-8b-prompt", kind="prompt", model="torirax-8b", dtype="bf16", position=0, tokens=2048),
        # latent and chunked attention, layers that loop
        dict(name="dumalix-1b-decode", kind="decode", model="dumalix-1b", dtype="bf16", position=4110, graph=True),
        # the next turn of a chat: a short portion after earlier ones
        dict(name="dumalix-1b-turn", kind="prompt", model="dumalix-1b", dtype="bf16", position=1500, tokens=61),
        # the largest: a full portion of the 8B class
        dict(name="dumalix-8b-prompt", kind="prompt", model="dumalix-8b", dtype="bf16", position=0, tokens=2048),
    ]


def draw(rng) -> dict:
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["llama decode", "llama batch", "llama prompt", "list decode", "list prompt", "list prompt"])
    if kind == "llama decode":
        model = rng.choice(["llama-1b", "llama-8b"])
        layers = rng.randint(4, 16) if model == "llama-8b" else 16
        most = 65001 if model == "llama-1b" else 16384
        return dict(kind="decode", model=model, layers=layers, position=spread(1, most), graph=rng.random() < 0.5)
    if kind == "llama batch":
        return dict(kind="batch", model="llama-8b", layers=4, sequences=spread(2, 64), longest=spread(512, 4096))
    if kind == "llama prompt":
        if rng.random() < 0.5:
            return dict(kind="prompt", model="llama-1b", layers=16, position=0, tokens=spread(2, 500))
        return dict(kind="prompt", model="llama-8b", layers=4, position=0, tokens=spread(2, 400))
    model = rng.choice(["torirax-1b", "dumalix-1b", "torirax-8b", "dumalix-8b"])
    dtype = "f32" if model.endswith("1b") and rng.random() < 0.3 else "bf16"
    if kind == "list decode":
        return dict(kind="decode", model=model, dtype=dtype, position=spread(2, 4096), graph=rng.random() < 0.5)
    most = 300 if dtype == "f32" else 2048
    return dict(kind="prompt", model=model, dtype=dtype, position=rng.choice([0, spread(2, 2000)]), tokens=spread(2, most))


# ---- weights: a tensor is given by the seed, its name and its shape --------------------------- #
def normal(seed: int, name: str, shape, std: float = 1.0, mean: float = 0.0) -> torch.Tensor:
    gen = torch.Generator(device="cuda").manual_seed(zlib.crc32(f"{seed} {name}".encode()))
    w = torch.empty(shape, device="cuda", dtype=torch.bfloat16).normal_(mean, std, generator=gen)
    return w


def token_ids(case: dict, seed: int, count: int, name: str) -> torch.Tensor:
    gen = torch.Generator(device="cuda").manual_seed(zlib.crc32(f"{seed} {name}".encode()))
    return torch.randint(0, VOCAB, (count,), generator=gen, device="cuda")


def llama_weights(case: dict, seed: int):
    """``get(name)`` of a llama case: matrices of one layer, embedding and head."""
    m = LLAMA[case["model"]]
    W, D, F = m["width"], m["dim"], m["ff"]
    shapes = {
        "qkv": ((m["heads"] + 2 * m["kv_heads"]) * D, W), "o": (W, m["heads"] * D), "up": (F, W), "gate": (F, W), "down": (W, F),
        "embed": (VOCAB, W), "head": (VOCAB, W),
    }

    def get(name: str, layer: int = -1) -> torch.Tensor:
        if name.startswith("norm"):
            return normal(seed, f"{layer} {name}", (W,), 0.1, 1.0)
        if name == "head" and m["tied"]:
            name = "embed"
        shape = shapes[name]
        std = shape[1] ** -0.5 / (math.sqrt(2 * case["layers"]) if name in ("o", "down") else 1.0)
        return normal(seed, f"{layer} {name}", shape, 0.1 if name == "embed" else std)

    return get


def list_config(case: dict) -> dict:
    """The ``config.json`` of a layer-list model with the widths of the llama models."""
    big = case["model"].endswith("8b")
    width, ff = (4096, 14336) if big else (2048, 8192)
    mlp = {"kind": "dense", "ff": ff}
    dim = 128 if big else 64
    layers = []
    if case["model"].startswith("torirax"):
        for group in range(6 if big else 5):
            layers += [{"type": "general_delta", "mixer": {"heads": width // 64, "dim": 64}, "mlp": mlp}] * 2
            mixer = {"heads": 16, "kv_heads": 4, "dim": dim, "vdim": 2 * dim, "scale": dim**-0.5, "diff": 0.5,
                     "mask": {"size": 2048 if big else 1024, "keep_first": 4}}
            if group % 2:  # every second one reads the keys of the one before it
                mixer["kv_from"] = len(layers) - 3
            layers.append({"type": "attention", "mixer": mixer, "mlp": mlp})
        return {"architecture": "Torirax", "width": width, "vocab": VOCAB, "max_positions": 8192, "norm": {"eps": 1e-5},
                "embedding": {"scale": width**0.5}, "layers": layers, "rank": 128 if big else 64}
    yarn = {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    latent = {"heads": 32 if big else 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192**-0.5,
              "rot": {"dims": 64, "base": 10000.0, "scaling": yarn}}
    chunked = {"heads": 32, "kv_heads": 8, "dim": dim, "vdim": dim, "scale": dim**-0.5, "mask": {"size": 8192}, "conv": 4,
               "rot": {"dims": dim, "base": 500000.0, "scaling": yarn}}
    mlp["limit"] = 7.0
    for i in range(24 if big else 12):
        layers.append({"type": "attention", "mixer": chunked, "mlp": mlp} if i % 2 else {"type": "latent_attention", "mixer": latent, "mlp": mlp})
    loop = {"start": 8, "stop": 12, "times": 3} if big else {"start": 4, "stop": 6, "times": 3}
    return {"architecture": "Dumalix", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5}, "canon": {"taps": 4}, "layers": layers,
            "loop": loop}


def list_shapes(cfg: dict) -> dict[str, tuple[int, ...]]:
    W, torirax = cfg["width"], cfg["architecture"] == "Torirax"
    out = {"embed": (VOCAB, W), "head": (VOCAB, W), "final.norm": (W,)}
    if torirax:
        out["pos"] = (cfg["max_positions"], W)
    else:
        out["loop.in"] = (W, 2 * W)
    for i, layer in enumerate(cfg["layers"]):
        m, p, mix = layer["mixer"], f"l{i}.", {}
        if layer["type"] == "general_delta":
            inner = m["heads"] * m["dim"]
            mix = {n: (inner, W) for n in "rkvag"} | {n: (inner,) for n in ("a.b", "w0", "norm")}
            mix |= {"w1": (cfg["rank"], W), "w2": (inner, cfg["rank"]), "o": (W, inner)}
        elif layer["type"] == "latent_attention":
            rank, H = m["kv_rank"], m["heads"]
            mix = {"q": (H * (m["dim"] + m["rot_dim"]), W), "dkv": (rank + m["rot_dim"], W), "dkv.norm": (rank,),
                   "uk": (H * m["dim"], rank), "uv": (H * m["vdim"], rank), "o": (W, H * m["vdim"])}
        else:
            maps = 2 if torirax else 1
            sizes = {"q": m["heads"] * maps * m["dim"], "k": m["kv_heads"] * maps * m["dim"], "v": m["kv_heads"] * m["vdim"]}
            mix = {n: (size, W) for n, size in sizes.items()} | {"o": (W, m["heads"] * m["vdim"])}
            if torirax:
                mix |= {n + ".b": (size,) for n, size in sizes.items()} | {"g": (m["heads"] * m["vdim"], W)}
                mix |= {n: (m["dim"],) for n in ("lq1", "lk1", "lq2", "lk2")}
            else:
                mix |= {n + ".conv": (size, m["conv"]) for n, size in sizes.items()}
                mix |= {"q.norm": (m["dim"],), "k.norm": (m["dim"],), "temp": (m["heads"],), "sink": (m["heads"],)}
        out |= {f"{p}mix.{n}": shape for n, shape in mix.items()}
        ff = layer["mlp"]["ff"]
        out |= {p + "norm1": (W,), p + "norm2": (W,), p + "mlp.up": (ff, W), p + "mlp.down": (W, ff)}
        out |= {p + "ls1": (W,), p + "ls2": (W,), p + "mlp.act": (4,)} if torirax else {p + "mlp.gate": (ff, W), p + "canon1": (W, 4)}
    return out


def list_weights(cfg: dict, seed: int):
    shapes = list_shapes(cfg)
    runs = len(layer_runs(cfg))
    offset = 0.0 if cfg["architecture"] == "Torirax" else 1.0  # (one-plus norms)

    def get(name: str) -> torch.Tensor:
        shape = shapes[name]
        if name.endswith(".conv") or name.endswith("canon1"):
            return normal(seed, name, shape, 0.2)
        if len(shape) == 2:
            std = 0.02 if name in ("embed", "pos") else shape[1] ** -0.5
            return normal(seed, name, shape, std / math.sqrt(2 * runs) if name.endswith((".o", ".down")) else std)
        if name.endswith(".act"):
            w = torch.tensor([0.6, 0.3, 0.2, 0.05], device="cuda")
            return (w + 0.05 * normal(seed, name, shape).float()).bfloat16()
        if name.endswith((".lq1", ".lk1", ".lq2", ".lk2", ".b", ".sink")):
            return normal(seed, name, shape, 0.1)
        if name.endswith(("norm1", "norm2", "final.norm")):
            return normal(seed, name, shape, 0.1, 1.0 - offset)
        return normal(seed, name, shape) if name.endswith(".w0") else normal(seed, name, shape, 0.1, 1.0)

    return get


# ---- prepare and run ------------------------------------------------------------------------- #
def lengths(case: dict) -> list[int]:
    """Ragged: spread over 256 .. ``longest`` (from half of it where it is small) out of order."""
    low = min(256, case["longest"] // 2)
    return [low + int((case["longest"] - low) * ((i + 1) * 0.6180339887 % 1.0)) for i in range(case["sequences"])]


def llama_model(case: dict, seed: int):
    m, get = LLAMA[case["model"]], llama_weights(case, seed)
    L = case["layers"]
    preset = LlamaConfig.llama_3_2_1b if case["model"] == "llama-1b" else LlamaConfig.llama_3_1_8b
    config = preset(num_hidden_layers=L)
    most = {"decode": case.get("position", 0) + 64, "batch": case.get("longest", 0) + 8, "prompt": case.get("position", 0) + case.get("tokens", 0) + 64}
    extra = ExtraModelConfig(interleave_rope=True, max_len_override=most[case["kind"]], max_batch_size=case.get("sequences", 1))

    def stack(name):
        first = get(name, 0)
        out = torch.empty((L, *first.shape), device="cuda", dtype=first.dtype)
        for i in range(L):
            out[i] = get(name, i)
        return out

    embed = get("embed")
    model = LlamaForCausalLM(
        config, extra, "cuda:0", torch.bfloat16, embed,
        StackedParams(qkv_proj=stack("qkv"), o_proj=stack("o"), attn_ln_weight=stack("norm1"), mlp_ln_weight=stack("norm2"),
                      up_proj=stack("up"), gate_proj=stack("gate"), down_proj=stack("down")),
        get("norm"), embed if m["tied"] else get("head"))
    return model


def llama_cache(case: dict, seed: int, layer: int, shape):
    return normal(seed, f"keys {layer}", shape), normal(seed, f"values {layer}", shape)


def prepare(case: dict, seed: int):
    torch.cuda.set_device(0)
    with torch.inference_mode():
        if case["model"] in LLAMA:
            model = llama_model(case, seed)
            k, v = model.stacked_kv_cache
            if case["kind"] != "prompt":
                for i in range(case["layers"]):
                    k[i], v[i] = llama_cache(case, seed, i, k[i].shape)
            B = case.get("sequences", 1)
            length = max(lengths(case)) if B > 1 else case["position"] + case.get("tokens", 0)
            parts = pick_num_attention_partitions(length, 64, model.device, model.num_kv_heads(), min_chunk_size=128)
            if B > 1:  # all sequences' partials of a layer in one wave
                parts = max(1, min(parts, 148 // (B * model.num_kv_heads())))
            gen = make_generator(model, LatencyScheduleOptions(
                num_attention_partitions=parts, coalesce_o_proj=True, merge_in_last_partial=True, batch_size=B))
        else:
            cfg = list_config(case)
            shapes, get = list_shapes(cfg), list_weights(cfg, seed)
            design = ToriraxForCausalLM if cfg["architecture"] == "Torirax" else DumalixForCausalLM
            extra = ExtraModelConfig(max_len_override=8192)
            model = design.assemble(design.read_config(cfg, shapes.__getitem__), extra, "cuda:0", DTYPES[case["dtype"]], get)
            gen = make_generator(model)
            if case["position"]:
                gen.feed(token_ids(case, seed, case["position"], "earlier"), 0, [])
        count = case.get("tokens", case.get("sequences", 1))
        tokens = token_ids(case, seed, count, "tokens")
        state = {"case": case, "gen": gen, "tokens": tokens.view(1, -1) if case["kind"] == "prompt" else tokens.view(-1, 1)}
        if case["kind"] == "batch":
            state["positions"] = lengths(case)
            state["rows"] = (torch.arange(count, device="cuda"), torch.tensor(state["positions"], device="cuda"))
        elif case["kind"] == "decode" and case["graph"]:
            if case["model"] not in LLAMA:
                # capturing runs nothing, so the recurrent state stays where the prompt left it
                gen.run(tokens[:1].view(1, 1), pos_id=case["position"] - 1)  # (first launches allocate)
                gen.feed(token_ids(case, seed, case["position"], "earlier"), 0, [])
            gen.enable_cuda_graph(warmup_pos=case["position"])
    return state


@torch.inference_mode()
def run(state):
    """Logits, and what the pass wrote into the sequences' state."""
    case, gen = state["case"], state["gen"]
    if case["model"] in LLAMA:
        k, v = gen.model.stacked_kv_cache
        if case["kind"] == "batch":
            gen.run(state["tokens"], state["positions"])
            return {"logits": gen.schedule.globs.logits, "keys": k[:, state["rows"][0], state["rows"][1]],
                    "values": v[:, state["rows"][0], state["rows"][1]]}
        if case["kind"] == "prompt":
            gen.prefill(state["tokens"])
        else:
            gen.run(state["tokens"], pos_id=case["position"])
        new = slice(case["position"], case["position"] + case.get("tokens", 1))
        return {"logits": gen.schedule.globs.logits, "keys": k[:, 0, new], "values": v[:, 0, new]}
    if case["kind"] == "prompt":
        logits = gen.feed(state["tokens"], case["position"], [case["tokens"] - 1])
    else:
        gen.run(state["tokens"], pos_id=case["position"])
        logits = gen.schedule.globs.logits.view(1, -1)
    held = gen.model.state
    new = slice(case["position"], case["position"] + case.get("tokens", 1))

    def rows(i, cache):
        if case["model"].startswith("dumalix") and cache.dim() == 4:
            return cache[0, :, new]  # by head
        where = held.rows[i]
        if where.total > new.stop:  # no row was used twice
            return cache[0, new]
        return cache[0, where.row(new.start) : where.row(new.start) + new.stop - new.start] if new.stop - new.start == 1 else cache[0]

    return {"logits": logits, "keys": [rows(i, c) for i, c in sorted(held.keys.items())],
            "values": [rows(i, c) for i, c in sorted(held.values.items())],
            "matrices": [c[0] for _, c in sorted(held.matrices.items())]}


# ---- what a pass cannot do without ------------------------------------------------------------ #
def work(case: dict) -> dict:
    """Weights once (once per run of a layer where layers loop), the keys that are seen, the rows,
    matrices and logits that are written; matrix products and attention."""
    n = case.get("tokens", 1)
    if case["model"] in LLAMA:
        m = LLAMA[case["model"]]
        W, D, L, B = m["width"], m["dim"], case["layers"], case.get("sequences", 1)
        params = L * (W * D * (2 * m["heads"] + 2 * m["kv_heads"]) + 3 * W * m["ff"])
        head = VOCAB * W
        seen = lengths(case) if B > 1 else [case["position"] + i for i in range(n)]
        row = 2 * m["kv_heads"] * D * L  # elements of a position's keys and values
        held = sum(seen) if B > 1 else seen[0]
        bytes_ = 2 * (params + head + 2 * L * W + (held + n * B) * row + n * B * W + B * VOCAB)
        flops = 2 * (n * B * params + B * head) + 4 * m["heads"] * D * L * sum(s + 1 for s in seen)
        return {"bytes": bytes_, "flops": flops}
    cfg = list_config(case)
    shapes = list_shapes(cfg)
    size = lambda name: math.prod(shapes[name])  # noqa: E731
    elem = 4 if case["dtype"] == "f32" else 2
    mats = lambda i: [x for x in shapes if x.startswith(f"l{i}.") and len(shapes[x]) == 2 and not x.endswith(("conv", "canon1"))]  # noqa: E731
    bytes_ = flops = 0.0
    at = range(case["position"], case["position"] + n)
    for i, enters in layer_runs(cfg):
        layer, m = cfg["layers"][i], cfg["layers"][i]["mixer"]
        params = sum(size(x) for x in mats(i) if not ("kv_from" in m and x.endswith(("mix.k", "mix.v"))))
        if enters:
            params += size("loop.in")
        bytes_ += elem * params
        flops += 2.0 * n * params
        if layer["type"] == "general_delta":
            state = m["heads"] * m["dim"] ** 2
            bytes_ += 8 * state
            flops += 10.0 * n * state
            continue
        if layer["type"] == "latent_attention":
            row, pair, most = m["kv_rank"] + m["rot_dim"], 2 * (m["dim"] + m["rot_dim"] + m["vdim"]), 1 << 30
        else:
            maps = 2 if cfg["architecture"] == "Torirax" else 1
            row, pair = m["kv_heads"] * (maps * m["dim"] + m["vdim"]), 2 * maps * (m["dim"] + m["vdim"])
            most = m["mask"]["size"] + m["mask"].get("keep_first", 0)
        bytes_ += elem * row * (min(at[0], most) + n)
        flops += pair * m["heads"] * sum(min(p + 1, most) for p in at)
    bytes_ += elem * (size("head") + n * cfg["width"]) + 4 * VOCAB
    flops += 2.0 * size("head")
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict):
    """Four times what two correct orders of summation and of rounding to the data type give."""
    if case.get("dtype") == "f32":
        return {"rel": 2e-5, "max": 5e-4}
    return {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits ------------------------------------------------------------------------ #
def rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def turn(x, angle, factor=1.0):
    """Neighbours (2i, 2i + 1) of the last axis turned by ``angle`` (broadcast against them)."""
    c, s = angle.cos() * factor, angle.sin() * factor
    n = 2 * angle.shape[-1]
    u, v = x[..., 0:n:2], x[..., 1:n:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2), x[..., n:]], dim=-1)


def attend(q, k, v, scale, mask, sink=None):
    """q [H, T, D], k [H, S, D], v [H, S, E]; ``mask`` [T, S]; a few heads at a time."""
    out = []
    for h in range(q.shape[0]):
        score = (q[h] @ k[h].T) * (scale[h] if torch.is_tensor(scale) else scale)
        score = score.masked_fill(~mask, float("-inf"))
        if sink is not None:
            score = torch.cat([score, sink[h].expand(score.shape[0], 1)], dim=1)
        p = torch.softmax(score, dim=-1)
        out.append(p[:, : k.shape[1]] @ v[h])
    return torch.stack(out)


def llama_frequencies(m: dict) -> torch.Tensor:
    D = m["dim"]
    f = 1.0 / (500000.0 ** (torch.arange(0, D, 2, dtype=torch.int64).float() / D))
    wave = 2 * math.pi / f
    smooth = (8192 / wave - 1.0) / (4.0 - 1.0)
    slow = torch.where(wave > 8192, f / m["factor"], f)
    mid = (1 - smooth) * slow / m["factor"] + smooth * slow
    return torch.where((wave <= 8192) & (wave >= 2048), mid, slow).double().cuda()


def llama_exact(case: dict, seed: int):
    m, get, eps = LLAMA[case["model"]], llama_weights(case, seed), 1e-5
    f64 = lambda name, i=-1: get(name, i).double()  # noqa: E731
    H, G, D, L, B = m["heads"], m["kv_heads"], m["dim"], case["layers"], case.get("sequences", 1)
    n = case.get("tokens", 1)
    ids = token_ids(case, seed, case.get("tokens", B), "tokens")
    seen = lengths(case) if B > 1 else [case["position"]]
    most = (case["longest"] + 8) if B > 1 else case["position"] + 64
    at = torch.tensor(seen, device="cuda") if B > 1 else torch.arange(case["position"], case["position"] + n, device="cuda")
    angle = at.double()[:, None, None] * llama_frequencies(m)
    x = get("embed")[ids].double()
    keys, values = [], []
    for i in range(L):
        h = rms(x, eps) * f64("norm1", i)
        q, k, v = (h @ f64("qkv", i).T).split([H * D, G * D, G * D], dim=-1)
        q, k, v = turn(q.view(-1, H, D), angle), turn(k.view(-1, G, D), angle), v.view(-1, G, D)
        keys.append(k)
        values.append(v)
        if case["kind"] == "prompt":
            mask = torch.ones(n, n, dtype=torch.bool, device="cuda").tril()
            a = attend(q.transpose(0, 1), k.transpose(0, 1).repeat_interleave(H // G, 0), v.transpose(0, 1).repeat_interleave(H // G, 0),
                       D**-0.5, mask).transpose(0, 1)
        else:
            kc, vc = llama_cache(case, seed, i, (B, most, G, D))
            rows = []
            for b, p in enumerate(seen):
                kk = torch.cat([kc[b, :p].double(), k[b : b + 1]]).transpose(0, 1)  # [G, p + 1, D]
                vv = torch.cat([vc[b, :p].double(), v[b : b + 1]]).transpose(0, 1)
                score = torch.softmax(q[b].view(G, H // G, D) @ kk.transpose(1, 2) * D**-0.5, dim=-1)
                rows.append((score @ vv).view(H, D))
            a = torch.stack(rows)
        x = x + a.reshape(-1, H * D) @ f64("o", i).T
        h = rms(x, eps) * f64("norm2", i)
        g = h @ f64("gate", i).T
        x = x + (g * torch.sigmoid(g) * (h @ f64("up", i).T)) @ f64("down", i).T
    last = x if B > 1 else x[-1:]
    logits = (rms(last, eps) * f64("norm")) @ f64("head").T
    return {"logits": logits if B > 1 else logits[0], "keys": torch.stack(keys), "values": torch.stack(values)}


def layer_runs(cfg: dict) -> list[tuple[int, bool]]:
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return [(i, False) for i in range(n)]
    a, b = loop["start"], loop["stop"]
    return [(i, False) for i in range(a)] + [(i, i == a) for i in range(a, b)] * loop["times"] + [(i, False) for i in range(b, n)]


def conv(u, w):
    """u [T, channels], w [channels, taps]; the last tap meets the current token."""
    taps, y = w.shape[1], u * w[:, -1]
    for back in range(1, min(taps, u.shape[0])):
        y[back:] += w[:, taps - 1 - back] * u[:-back]
    return y


def frequencies(rot: dict):
    i = torch.arange(rot["dims"] // 2, dtype=torch.float64, device="cuda")
    f = rot["base"] ** (-2.0 * i / rot["dims"])
    y = rot["scaling"]
    place = lambda turns: rot["dims"] * math.log(y["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))  # noqa: E731
    lo, hi = max(math.floor(place(y["fast"])), 0), min(math.ceil(place(y["slow"])), rot["dims"] - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / y["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(y["factor"]) + 1


def delta_exact(h, W, m, eps):
    """Output and the last state [heads, value, key]."""
    T, H, D = h.shape[0], m["heads"], m["dim"]
    r, k, v = ((h @ W(n).T).view(T, H, D) for n in "rkv")
    w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ W("w1").T) @ W("w2").T + W("w0"))).view(T, H, D)
    a = torch.sigmoid(h @ W("a").T + W("a.b")).view(T, H, D)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S = torch.zeros(H, D, D, dtype=h.dtype, device=h.device)  # [value, key]
    out = torch.empty_like(r)
    au = a * u
    for t in range(T):
        read = S @ u[t].unsqueeze(-1)
        S = S * w[t].unsqueeze(1)
        S.baddbmm_(torch.cat([read, v[t].unsqueeze(-1)], dim=-1), torch.stack([-au[t], k[t]], dim=1))
        out[t] = (S @ r[t].unsqueeze(-1)).squeeze(-1)
    o = rms(out, eps).reshape(T, H * D) * W("norm") * torch.sigmoid(h @ W("g").T)
    return o @ W("o").T, S


def list_exact(case: dict, seed: int):
    cfg = list_config(case)
    get, eps, width = list_weights(cfg, seed), cfg["norm"]["eps"], cfg["width"]
    W = lambda name: get(name).double()  # noqa: E731
    torirax = cfg["architecture"] == "Torirax"
    ids = token_ids(case, seed, case.get("tokens", 1), "tokens")
    if case["position"]:
        ids = torch.cat([token_ids(case, seed, case["position"], "earlier"), ids])
    T, first = ids.numel(), case["position"]
    at = torch.arange(T, device="cuda")
    causal = at[:, None] >= at[None, :]
    x = get("embed")[ids].double()
    if torirax:
        x = x * cfg["embedding"]["scale"] + get("pos")[:T].double()
    start = x
    keys, values, matrices, own = [], [], [], {}
    for i, enters in layer_runs(cfg):
        layer, p = cfg["layers"][i], f"l{i}."
        m, M = layer["mixer"], lambda name, p=p: W(f"{p}mix.{name}")
        if enters:
            x = torch.cat([x, start], dim=-1) @ W("loop.in").T
        if torirax:
            norm = lambda y, w: rms(y - y.mean(-1, keepdim=True), eps) * w  # noqa: E731
        else:
            norm = lambda y, w: rms(y, eps) * (1 + w)  # noqa: E731
        h = norm(x, W(p + "norm1"))
        if not torirax:
            h = h + conv(h, W(p + "canon1"))
        if layer["type"] == "general_delta":
            y, S = delta_exact(h, M, m, eps)
            matrices.append(S)
        elif layer["type"] == "latent_attention":
            H, D, R, E, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            q, down = (h @ M("q").T).view(T, H, D + R), h @ M("dkv").T
            c = rms(down[:, :rank], eps) * M("dkv.norm")
            f, factor = frequencies(m["rot"])
            angle = at.double()[:, None] * f
            shared = turn(down[:, rank:], angle, factor)
            q = torch.cat([q[..., :D], turn(q[..., D:], angle[:, None], factor)], dim=-1).transpose(0, 1)
            k = torch.cat([(c @ M("uk").T).view(T, H, D), shared[:, None].expand(T, H, R)], dim=-1).transpose(0, 1)
            y = attend(q, k, (c @ M("uv").T).view(T, H, E).transpose(0, 1), m["scale"], causal).transpose(0, 1).reshape(T, H * E) @ M("o").T
            keys.append(None)  # (latent rows: a layout of their own)
        elif torirax:
            H, G, D, E = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q = (h @ M("q").T + M("q.b")).view(T, H, 2, D)
            if "kv_from" in m:
                k, v = own[m["kv_from"]]
            else:
                k, v = own[i] = (h @ M("k").T + M("k.b")).view(T, G, 2, D), (h @ M("v").T + M("v.b")).view(T, G, E)
                whole = min(8192, m["mask"]["size"] + 2048 + m["mask"]["keep_first"]) > T  # a row per position
                keys.append(k[first:] if whole else None)
                values.append(v[first:] if whole else None)
            mask = causal & ((at[:, None] - at[None, :] < m["mask"]["size"]) | (at[None, :] < m["mask"]["keep_first"]))
            spread = lambda y: y.transpose(0, 1).repeat_interleave(H // G, 0)  # noqa: E731
            a = [attend(q[:, :, j].transpose(0, 1), spread(k[:, :, j]), spread(v), m["scale"], mask) for j in (0, 1)]
            lam = torch.exp((M("lq1") * M("lk1")).sum()) - torch.exp((M("lq2") * M("lk2")).sum()) + m["diff"]
            o = (rms(a[0] - lam * a[1], eps) * (1 - m["diff"])).transpose(0, 1).reshape(T, H * E)
            y = (o * torch.sigmoid(h @ M("g").T)) @ M("o").T
        else:
            H, G, D, E = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q, k, v = (conv(h @ M(n).T, M(n + ".conv")) for n in "qkv")
            f, factor = frequencies(m["rot"])
            angle = at.double()[:, None, None] * f
            plain = at.double()[:, None, None] * m["rot"]["base"] ** (-2.0 * torch.arange(E // 2, dtype=torch.float64, device="cuda") / E)
            q = turn(rms(q.view(T, H, D), eps) * M("q.norm"), angle, factor)
            k = turn(rms(k.view(T, G, D), eps) * M("k.norm"), angle, factor)
            v = turn(v.view(T, G, E), plain)
            keys.append(k[first:].transpose(0, 1))
            values.append(v[first:].transpose(0, 1))
            mask = causal & (at[:, None] // m["mask"]["size"] == at[None, :] // m["mask"]["size"])
            spread = lambda y: y.transpose(0, 1).repeat_interleave(H // G, 0)  # noqa: E731
            o = attend(q.transpose(0, 1), spread(k), spread(v), m["scale"] * M("temp"), mask, M("sink"))
            y = turn(o.transpose(0, 1), -plain).reshape(T, H * E) @ M("o").T
        if torirax:
            x = x + y * W(p + "ls1")
            z = norm(x, W(p + "norm2")) @ W(p + "mlp.up").T
            a, b, c, e = W(p + "mlp.act")
            z = a * rms(z, eps) + b * rms(z**2, eps) + c * rms(z**3, eps) + e
            x = x + (z @ W(p + "mlp.down").T) * W(p + "ls2")
        else:
            z = norm(x, W(p + "norm2"))
            g = (z @ W(p + "mlp.gate").T).clamp(max=7.0)
            u = (z @ W(p + "mlp.up").T).clamp(-7.0, 7.0)
            x = x + y + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ W(p + "mlp.down").T
    x = x[-1:]
    x = norm(x, W("final.norm"))
    return {"logits": x @ W("head").T, "keys": keys, "values": values, "matrices": matrices}


@torch.inference_mode()
def exact(case: dict, seed: int):
    torch.cuda.set_device(0)
    return llama_exact(case, seed) if case["model"] in LLAMA else list_exact(case, seed)
