"""The inferences this framework is used for, as cases that can be timed.

A case is one compiled module (a model family at a batch and a length) and one way of calling it,
or one call of the stand-alone attention. Models keep their full widths and depths throughout; what
varies is what varies between requests: how many there are, how long they are, how much of them is
padding, and whether the program keeps its tensors on the host or on the device.

``io`` is how the program calls a module:
  host    the prepared host runner: pinned inputs are copied in, one launch, the outputs are copied
          to pinned memory and waited for. What a server does that answers single requests.
  device  inputs and outputs are device tensors of the program: copied to the module's parameters,
          one launch, the outputs copied out, nothing waited for. What a pipeline does that goes on
          on the GPU (throughput jobs, a sampler behind the logits).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from mononn_b200 import compile_encoder, compile_hlo
from mononn_b200.hlo_builder import bert_hlo, clip_hlo, opt_hlo, t5_hlo, vit_hlo
from mononn_b200.models import (EncoderConfig, T5_BUCKETS, bert_base, bert_weight_shapes, clip_b32,
                                clip_weight_shapes, opt_1p3b, opt_weight_shapes, t5_position_bias, t5_small,
                                t5_weight_shapes, vit_weight_shapes)
from mononn_b200.module import attention_noalloc

LARGEST_FLOPS = 3.95e12  # 24 layers, width 1024, 16 sequences of 384


def listed() -> list[dict]:
    return [
        # the attention of one layer for a host that owns the device memory: a single sequence
        {"name": "attention_b1_s128", "family": "attention", "batch": 1, "heads": 12, "seq": 128, "pad": 0.25,
         "causal": False},
        # a search query of a few words
        {"name": "bert_base_b1_s24", "family": "bert", "batch": 1, "seq": 24, "pad": 0.0, "io": "host",
         "frontend": "hlo"},
        # the headline: one request, one passage
        {"name": "bert_base_b1_s128", "family": "bert", "batch": 1, "seq": 128, "pad": 0.0, "io": "host",
         "frontend": "hlo"},
        # a few requests of odd length batched together, padded to the longest
        {"name": "bert_base_b8_s100", "family": "bert", "batch": 8, "seq": 100, "pad": 0.3, "io": "device",
         "frontend": "hlo"},
        # question answering over one long passage
        {"name": "bert_large_b1_s384", "family": "bert_large", "batch": 1, "seq": 384, "pad": 0.25, "io": "host",
         "frontend": "hlo"},
        # the same offline, batched: the largest job
        {"name": "bert_large_b16_s384", "family": "bert_large", "batch": 16, "seq": 384, "pad": 0.25,
         "io": "device", "frontend": "builder"},
        # one image, 197 tokens
        {"name": "vit_base_b1", "family": "vit", "batch": 1, "image": 224, "io": "host"},
        # a batch of images already on the GPU
        {"name": "vit_base_b64", "family": "vit", "batch": 64, "image": 224, "io": "device"},
        # prefill of one prompt, and of eight, with logits of every position for what samples next
        {"name": "opt_1p3b_b1_s128", "family": "opt", "batch": 1, "seq": 128, "io": "device"},
        {"name": "opt_1p3b_b8_s128", "family": "opt", "batch": 8, "seq": 128, "io": "device"},
        # images against texts, both towers in one launch
        {"name": "clip_b32_i32_t32", "family": "clip", "images": 32, "texts": 32, "io": "host"},
        # encoder and decoder of one sequence pair
        {"name": "t5_small_b1_s128", "family": "t5", "batch": 1, "seq": 128, "io": "host"},
    ]


def _log(rng, low: int, high: int) -> int:
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng) -> dict:
    while True:
        family = rng.choices(["bert", "bert_large", "vit", "opt", "clip", "t5", "attention"],
                             [6, 2, 3, 2, 2, 2, 3])[0]
        io = rng.choice(["host", "device"])
        pad = rng.choice([0.0, round(rng.uniform(0.05, 0.5), 2)])
        if family == "attention":
            seq = _log(rng, 8, 128)
            c = {"family": family, "batch": _log(rng, 1, min(128, 16384 // seq)), "heads": rng.choice([8, 12, 16]),
                 "seq": seq, "pad": pad, "causal": rng.random() < 0.3}
        elif family in ("bert", "bert_large"):
            c = {"family": family, "batch": _log(rng, 1, 32), "seq": _log(rng, 8, 384), "pad": pad, "io": io,
                 "frontend": rng.choice(["hlo", "builder"])}
            if c["batch"] * c["seq"] > (4096 if c["frontend"] == "hlo" else 6144):
                continue
        elif family == "vit":
            c = {"family": family, "batch": _log(rng, 1, 48), "image": rng.choice([160, 192, 224]), "io": io}
        elif family == "opt":
            c = {"family": family, "batch": _log(rng, 1, 8), "seq": _log(rng, 8, 256), "io": io}
            if c["batch"] * c["seq"] > 1024:
                continue
        elif family == "clip":
            c = {"family": family, "images": _log(rng, 1, 48), "texts": _log(rng, 1, 48), "io": io}
        else:
            c = {"family": family, "batch": _log(rng, 1, 16), "seq": rng.choice([32, 64, 96, 128]), "io": io}
        if work(c)["flops"] <= LARGEST_FLOPS:
            return c


# ------------------------------------------------------------------------------------- modules
def _config(case: dict):
    family, batch = case["family"], case.get("batch", 1)
    if family == "bert":
        return bert_base(batch, case["seq"])
    if family == "bert_large":
        return EncoderConfig(layers=24, hidden=1024, heads=16, ffn=4096, batch=batch, seq=case["seq"])
    if family == "vit":
        n = (case["image"] // 16) ** 2 + 1
        return EncoderConfig(model="vit", batch=batch, seq=n, image=case["image"], patch=16, channels=3, max_pos=n,
                             vocab=0, types=0)
    if family == "opt":
        return opt_1p3b(batch, case["seq"])
    if family == "clip":
        return clip_b32(case["images"], case["texts"])
    return t5_small(batch, case["seq"])


def _shapes(cfg) -> dict[str, tuple[int, ...]]:
    return {"bert": bert_weight_shapes, "vit": vit_weight_shapes, "opt": opt_weight_shapes,
            "clip": clip_weight_shapes, "t5": t5_weight_shapes}[cfg.model](cfg)


def _weights(cfg) -> dict[str, np.ndarray]:
    """Random-init weights N(0, 0.02), biases and norm shifts too, norm scales around 1. The token
    table of the decoder is drawn wider: its logits then have a leader, as a trained model's do,
    where 50272 near-equal ones would leave the arg-max to the rounding of the last bit."""
    gen = torch.Generator(device="cuda").manual_seed(1234)
    out = {}
    for name, shape in _shapes(cfg).items():
        std = 1.0 if cfg.model == "opt" and name == "embeddings.word" else 0.02
        w = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * std
        if name.endswith(".gamma"):
            w += 1.0
        if name.endswith(".rel_bias"):
            stack, s = name.split(".")[0], cfg.seq
            assert shape == (T5_BUCKETS, cfg.heads)
            bias = t5_position_bias(w.cpu().numpy(), s, s, stack == "encoder")
            out[stack + ".pos_bias"] = bias.reshape(cfg.heads * s, s).astype(np.float16)
        else:
            out[name] = w.half().cpu().numpy()
    return out


@functools.lru_cache(maxsize=20)
def _module(key: tuple):
    """The module that a program compiles once and keeps for all its requests of a shape."""
    case = dict(key)
    cfg = _config(case)
    weights = _weights(cfg)
    if case.get("frontend") == "builder":
        mod, names = compile_encoder(cfg), {k: k for k in weights}
    else:
        hlo = {"bert": bert_hlo, "vit": vit_hlo, "opt": opt_hlo, "clip": clip_hlo, "t5": t5_hlo}[cfg.model]
        text, names = hlo(cfg)
        mod = compile_hlo(text)
    for name, value in weights.items():
        mod.set_constant(names[name], value)
    mod.allocate()
    return mod


def _inputs(cfg, case: dict, gen) -> list[torch.Tensor]:
    """Device tensors by parameter number: ids uniform over the vocabulary, pixels in [-1, 1]."""
    def ids(c):
        return torch.randint(0, c.vocab, (c.batch, c.seq), generator=gen, device="cuda", dtype=torch.int32)

    def pixels(c):
        return torch.rand((c.batch, c.channels, c.image, c.image), generator=gen, device="cuda") * 2.0 - 1.0

    if cfg.model == "bert":
        return [ids(cfg), _mask(cfg.batch, cfg.seq, case["pad"], gen),
                torch.zeros((cfg.batch, cfg.seq), dtype=torch.int32, device="cuda")]
    if cfg.model == "vit":
        return [pixels(cfg)]
    if cfg.model == "opt":
        return [ids(cfg)]
    if cfg.model == "clip":
        return [pixels(cfg.vision), ids(cfg.text)]
    return [ids(cfg), ids(cfg)]


def _mask(batch: int, seq: int, pad: float, gen) -> torch.Tensor:
    """Every sequence ends in up to twice `pad` of padding; one of them is full."""
    lost = (torch.rand(batch, generator=gen, device="cuda") * 2.0 * pad * seq).long().clamp(max=seq - 1)
    lost[0] = 0 if batch > 1 else int(pad * seq)
    return (torch.arange(seq, device="cuda")[None, :] < (seq - lost)[:, None]).int().contiguous()


def _outputs(cfg) -> list[tuple[torch.dtype, tuple[int, ...]]]:
    if cfg.model == "opt":
        return [(torch.float16, (cfg.tokens, cfg.vocab)), (torch.int32, (cfg.tokens,))]
    if cfg.model == "clip":
        ni, nt = cfg.vision.batch, cfg.text.batch
        return [(torch.float16, (ni, nt)), (torch.float16, (ni, cfg.proj)), (torch.float16, (nt, cfg.proj))]
    return [(torch.float16, (cfg.tokens, cfg.hidden))]


def _bytes(t: torch.Tensor) -> torch.Tensor:
    return t.reshape(-1).view(torch.uint8)


# ------------------------------------------------------------------------------- prepare and run
def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["family"] == "attention":
        b, h, s = case["batch"], case["heads"], case["seq"]
        pitch = (s + 7) // 8 * 8  # rows of the transposed values start on 16 bytes
        q, k = (torch.randn((b * s, h * 64), generator=gen, device="cuda").half() for _ in range(2))
        vt = torch.zeros((b * h * 64, pitch), dtype=torch.float16, device="cuda")
        vt[:, :s] = torch.randn((b * h * 64, s), generator=gen, device="cuda").half()
        mask = _mask(b, s, case["pad"], gen) if case["pad"] else None
        return {"q": q, "k": k, "vt": vt, "mask": mask, "out": torch.empty_like(q), "case": case}

    cfg = _config(case)
    mod = _module(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "pad", "io"))))
    inputs = _inputs(cfg, case, gen)
    state = {"io": case["io"], "module": mod}
    if case["io"] == "host":
        host_in = [t.cpu().pin_memory() for t in inputs]
        host_out = [torch.empty(shape, dtype=dtype).pin_memory() for dtype, shape in _outputs(cfg)]
        state.update(outputs=host_out, call=mod.host_runner(host_in, host_out))
    else:
        descs, bufs = mod.args(), mod.buffers
        outputs = [torch.empty(shape, dtype=dtype, device="cuda") for dtype, shape in _outputs(cfg)]

        def moves(kind, tensors):  # (buffer of the module, tensor of the program) for each argument
            at = [(bufs[d["index"]], _bytes(tensors[d["param_number"]])) for d in descs if d["kind"] == kind]
            return [(b[: t.numel()], t) for b, t in at]

        state.update(outputs=outputs, copy_in=moves(0, inputs), copy_out=moves(1, outputs))
    return state


def run(state: dict):
    if "q" in state:
        c = state["case"]
        b, h, s = c["batch"], c["heads"], c["seq"]
        mask = state["mask"]
        attention_noalloc(state["q"].data_ptr(), state["k"].data_ptr(), state["vt"].data_ptr(),
                          None if mask is None else mask.data_ptr(), state["out"].data_ptr(), b, h, s, h * 64,
                          state["vt"].shape[1], h * 64, 1.0 / 8.0, causal=c["causal"])
        return state["out"]
    if state["io"] == "host":
        state["call"]()
        return state["outputs"]
    for param, tensor in state["copy_in"]:
        param.copy_(tensor)
    state["module"].launch()
    for live_out, tensor in state["copy_out"]:
        tensor.copy_(live_out)
    return state["outputs"]


# ------------------------------------------------------------------------------ work and tolerance
def _block_flops(t: int, batch: int, seq: int, h: int, f: int) -> float:
    """One transformer block: four projections, scores and context, the two FFN products."""
    return 2.0 * t * (4 * h * h + 2 * h * f) + 4.0 * batch * seq * seq * h


def work(case: dict) -> dict:
    if case["family"] == "attention":
        b, h, s = case["batch"], case["heads"], case["seq"]
        return {"bytes": 4.0 * b * s * h * 64 * 2 + (4.0 * b * s if case["pad"] else 0.0),
                "flops": 4.0 * b * h * s * s * 64}
    cfg = _config(case)
    v, t = (cfg.vision, cfg.text) if cfg.model == "clip" else (cfg, cfg)
    moved = 0.0
    for name, shape in _shapes(cfg).items():
        n = float(math.prod(shape))
        leaf = name.removeprefix("vision.").removeprefix("text.")
        if leaf in ("embeddings.word", "shared") and cfg.model != "opt":  # only the rows that are looked up
            n = min(n, float(t.tokens * t.hidden * (2 if cfg.model == "t5" else 1)))
        elif leaf == "embeddings.position" and cfg.model in ("bert", "opt"):
            n = float(cfg.seq * cfg.hidden)
        elif leaf.endswith("rel_bias"):
            n = float(cfg.heads * cfg.seq * cfg.seq)
        moved += 2.0 * n
    if cfg.model in ("vit", "clip"):
        moved += 4.0 * v.batch * v.channels * v.image * v.image
    if cfg.model != "vit":
        moved += 4.0 * t.tokens * {"bert": 3, "t5": 2}.get(cfg.model, 1)
    moved += sum((2.0 if dtype == torch.float16 else 4.0) * math.prod(shape) for dtype, shape in _outputs(cfg))

    flops = t.layers * _block_flops(t.tokens, t.batch, t.seq, t.hidden, t.ffn)
    if cfg.model == "clip":
        flops += v.layers * _block_flops(v.tokens, v.batch, v.seq, v.hidden, v.ffn)
        flops += 2.0 * cfg.proj * (v.batch * v.hidden + t.batch * t.hidden + v.batch * t.batch)
    if cfg.model in ("vit", "clip"):
        flops += 2.0 * v.batch * (v.seq - 1) * v.hidden * v.channels * v.patch * v.patch
    if cfg.model == "opt":
        flops += 2.0 * t.tokens * t.hidden * t.vocab
    if cfg.model == "t5":  # the decoder: the same blocks and a cross-attention each
        flops += flops + t.layers * (8.0 * t.tokens * t.hidden ** 2 + 4.0 * t.batch * t.seq ** 2 * t.hidden)
    return {"bytes": moved, "flops": flops}


def tolerance(case: dict) -> dict:
    """f16 storage between operators, f32 sums: each stored tensor is off by 2^-11 / sqrt(3) = 2.8e-4
    of its value. One attention stores its probabilities and its result; a model stores about ten
    tensors a layer, whose errors add up in quadrature over 12 to 24 layers to some 4e-3 (less where a
    residual stream is kept in f32). The token ids follow the logits."""
    if case["family"] == "attention":
        return {"rel": 1e-3, "max": 1e-2}
    return {"rel": 5e-3, "max": 5e-2, "differ": 0.005}
