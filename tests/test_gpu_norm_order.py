"""A norm does not depend on how many warps share its rows (-m gpu). The embedding's LayerNorm gives each
row to one warp; the same rows through the norm of a layer, where two warps share rows of 513 to 1024
columns, have to come out the same, bit for bit."""
import dataclasses

import numpy as np
import pytest

from mononn_b200 import bert_tiny, compile_hlo
from mononn_b200.hlo_builder import bert_hlo
from mononn_b200.models import bert_weight_shapes
from tests.test_gpu_parity import run_module

pytestmark = pytest.mark.gpu

TRIALS = 64


def build(cfg, weights):
    text, names = bert_hlo(cfg)
    mod = compile_hlo(text, barrier_timeout_us=500000)
    mod.set_weights({names[k]: weights[k] for k in bert_weight_shapes(cfg)})
    return mod, names


def run(mod, cfg, ids):
    return run_module(mod, cfg, {"input_ids": ids, "attention_mask": np.ones_like(ids), "token_type_ids": 0 * ids})


@pytest.mark.parametrize("hidden", [512, 576, 768, 832, 1024])
def test_rows_shared_by_two_warps_equal_rows_of_one(hidden):
    """A layer whose matrices and first scale are zero hands its first shift to its last norm, in every
    row; an embedding without layers hands each row of its table to the same norm."""
    rows, seq = 400, 40  # more rows than are dealt to four warps each
    cfg = bert_tiny(batch=rows // seq, seq=seq, layers=1, hidden=hidden, ffn=64)
    rng = np.random.default_rng(hidden)
    values = rng.normal(0.1, 1.0, (TRIALS, hidden)).astype(np.float16)
    scale, shift = (rng.normal(m, 0.3, hidden).astype(np.float16).astype(np.float32) for m in (1.0, 0.0))
    w = {k: np.zeros(s, np.float32) for k, s in bert_weight_shapes(cfg).items()}
    w["layer0.ffn.ln.gamma"], w["layer0.ffn.ln.beta"] = scale, shift
    mod, names = build(cfg, w)
    norms = [o for s in mod.plan()["stages"] for o in s["ops"] if o["kind"] == "layernorm"]
    assert len(norms) == 2 and all(o["n_items"] == rows // 8 for o in norms)  # eight rows an item: not dealt to four

    one = dataclasses.replace(cfg, layers=0, batch=1, seq=TRIALS, vocab=TRIALS, max_pos=TRIALS)
    w1 = {k: np.zeros(s, np.float32) for k, s in bert_weight_shapes(one).items()}
    w1["embeddings.word"] = values.astype(np.float32)
    w1["embeddings.ln.gamma"], w1["embeddings.ln.beta"] = scale, shift
    mod1, _ = build(one, w1)
    want = run(mod1, one, np.arange(TRIALS, dtype=np.int32)[None, :])
    mod1.close()

    off = 0
    for i in range(TRIALS):
        mod.set_constant(names["layer0.attn.ln.beta"], values[i])
        got = run(mod, cfg, np.zeros((cfg.batch, seq), np.int32))
        off += int((got != want[i]).any(axis=0).sum())
    mod.close()
    assert off == 0, f"{off} of {TRIALS * hidden} values differ"
