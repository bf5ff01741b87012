"""Stages in which a CTA works on two norms whose rows are shared by warps: the warps of a row show each
other their sums in shared memory, and the second norm's must not land where a slower warp still
reads the first's."""
import pytest

from mononn_b200 import clip_tiny, make_t5_inputs, make_weights, t5_tiny
from mononn_b200.hlo_builder import clip_hlo, t5_hlo
from mononn_b200.module import describe
from oracle import ref_encoder as R
from tests.helpers import assert_parity
from tests.test_gpu_parity import check_clip, run_t5

ROW_SPLIT = 1 << 14
CASES = {
    "t5": t5_tiny(batch=2, seq=128, layers=1, hidden=512, ffn=64),
    "clip": clip_tiny(images=4, texts=3, image=224, layers=2, vh=768, th=512, seq=77, vocab=1000),
    "clip_few_texts": clip_tiny(images=24, texts=3, image=96, layers=1, vh=768, th=512, seq=77, vocab=1000),
}


def two_norms_on_a_cta(plan, grid=148):
    """Stages in which some CTA has items of two such norms."""
    found = 0
    for stage in plan["stages"]:
        base, seen, twice = 0, set(), False
        for op in stage["ops"]:
            ctas = {i % grid for i in range(base, base + op["n_items"])}
            base += op["n_items"]
            if op["kind"] == "layernorm" and op["flags"] & ROW_SPLIT:
                twice = twice or bool(ctas & seen)
                seen |= ctas
        found += twice
    return found


@pytest.mark.parametrize("name", sorted(CASES))
def test_the_cases_have_such_stages(name):
    cfg = CASES[name]
    text, _ = (t5_hlo if cfg.model == "t5" else clip_hlo)(cfg)
    assert two_norms_on_a_cta(describe("hlo", text)["plan"]) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_two_norms_on_a_cta_against_the_oracle(name):
    cfg = CASES[name]
    for seed in (71, 72, 73):
        if cfg.model == "clip":
            check_clip(cfg, seed)
        else:
            w, inp = make_weights(cfg, seed, stress=True), make_t5_inputs(cfg, seed)
            assert_parity(run_t5(cfg, w, inp), R.t5_model(cfg, w, inp), "T5")
