"""LayerNorm rows at the edges of how they are dealt to warps (-m gpu): one, two and four warps to a
row (512 columns a warp), more rows than one round of the CTAs takes, and a last item that is not full."""
import pytest

from mononn_b200 import bert_tiny, make_inputs, make_weights
from oracle import ref_encoder as R
from tests.helpers import assert_parity
from tests.test_gpu_parity import build, run_module

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch, seq, hidden", [
    (1, 3, 1088),     # four warps to a row, two rows an item, an odd last row
    (37, 8, 64),      # 296 rows: the most that are shared by four warps
    (9, 33, 512),     # 297 rows: one warp to a row, 512 columns: all its vectors in use
    (9, 33, 576),     # two warps to a row, 288 columns each
    (5, 61, 1024),    # two warps to a row, full
    (3, 101, 1088),   # four warps to a row because it is wide: 303 rows in items of eight
    (40, 64, 64),     # 2560 rows: three items and more for a CTA
    (47, 64, 576),    # 3008 rows of two warps each: an odd number of steps for some CTAs
], ids=lambda v: str(v))
def test_layernorm_rows_at_the_edges(batch, seq, hidden):
    cfg = bert_tiny(batch=batch, seq=seq, layers=1, hidden=hidden, ffn=64)
    w = make_weights(cfg, 91, stress=True)
    inp = make_inputs(cfg, 91)
    mod = build(cfg, w, "hlo")
    got = run_module(mod, cfg, inp)
    mod.close()
    assert_parity(got, R.bert_encoder(cfg, w, inp), f"{batch * seq} rows of {hidden}")
