"""Norm rows at the edges of how they are dealt to warps (-m gpu): one, two and four warps to a row (512
columns a warp), more rows than one round of the CTAs takes, and a last item that is not full; for
LayerNorm, RMS norm and L2 norm, from f16 and f32 rows."""
import pytest

from mononn_b200 import (bert_tiny, clip_tiny, make_inputs, make_t5_inputs, make_vit_inputs, make_weights, t5_tiny,
                         vit_tiny)
from oracle import ref_encoder as R
from tests.helpers import assert_parity
from tests.test_gpu_parity import build, check_clip, run_module, run_t5, run_vit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch, seq, hidden", [
    (1, 3, 1088),     # four warps to a row, two rows an item, an odd last row
    (37, 8, 64),      # 296 rows: the most that are shared by four warps
    (9, 33, 512),     # 297 rows: one warp to a row, 512 columns: all its vectors in use
    (9, 33, 576),     # two warps to a row, 288 columns each
    (5, 61, 1024),    # two warps to a row, full
    (3, 101, 1088),   # four warps to a row because it is wide: 303 rows in items of eight
    (40, 64, 64),     # 2560 rows: two or three items for a CTA
    (47, 64, 576),    # 3008 rows of two warps each: two or three items of two steps for a CTA
    (1, 3, 2048),     # four warps to a row, 512 columns each: all their vectors in use, an odd last row
    (3, 101, 2048),   # the same because it is wide, in items of eight
], ids=lambda v: str(v))
def test_layernorm_rows_at_the_edges(batch, seq, hidden):
    cfg = bert_tiny(batch=batch, seq=seq, layers=1, hidden=hidden, ffn=64)
    w = make_weights(cfg, 91, stress=True)
    inp = make_inputs(cfg, 91)
    mod = build(cfg, w, "hlo")
    got = run_module(mod, cfg, inp)
    mod.close()
    assert_parity(got, R.bert_encoder(cfg, w, inp), f"{batch * seq} rows of {hidden}")


@pytest.mark.parametrize("batch, hidden", [
    (1, 2048),   # 32 rows, four warps to a row, full
    (10, 512),   # 320 rows: one warp to a row
    (10, 576),   # two warps, 384 and 192 columns
    (10, 1024),  # two warps, full
    (10, 1088),  # four warps, in items of eight
], ids=lambda v: str(v))
def test_rms_norm_rows(batch, hidden):
    cfg = t5_tiny(batch=batch, seq=32, layers=1, hidden=hidden, ffn=64)
    w, inp = make_weights(cfg, 92, stress=True), make_t5_inputs(cfg, 92)
    assert_parity(run_t5(cfg, w, inp), R.t5_model(cfg, w, inp), f"{batch * 32} RMS rows of {hidden}")


@pytest.mark.parametrize("images, proj", [
    (5, 2048),    # four warps to a row, full; odd rows of the class tokens (every other source row)
    (300, 512),   # one warp to a row
    (300, 832),   # two warps, 512 and 320 columns
    (300, 1088),  # four warps, in items of eight
], ids=lambda v: str(v))
def test_l2_norm_rows(images, proj):
    check_clip(clip_tiny(images=images, texts=3, image=32, patch=32, proj=proj), 93)


@pytest.mark.parametrize("batch, hidden", [
    (60, 576),   # 300 rows: two warps
    (60, 1088),  # four warps
    (3, 1088),   # 15 rows dealt to four warps each
], ids=lambda v: str(v))
def test_rows_of_an_f32_stream(batch, hidden):
    cfg = vit_tiny(batch=batch, image=32, patch=16, layers=1, hidden=hidden)
    w, inp = make_weights(cfg, 94, stress=True), make_vit_inputs(cfg, 94)
    assert_parity(run_vit(cfg, w, inp), R.vit_encoder(cfg, w, inp), f"{batch * 5} f32 rows of {hidden}")
