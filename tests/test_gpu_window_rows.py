"""Window rows of a convolution at the edges of their batches (-m gpu): a lane has eight pixels of a row
in flight (256 columns); rows that end inside a batch, at its end, and one group after it."""
import numpy as np
import pytest

from mononn_b200 import make_vit_inputs, make_weights, vit_tiny
from oracle import ref_encoder as R
from tests.helpers import assert_parity
from tests.test_gpu_parity import run_vit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("image, patch, stride, pad", [
    (12, 4, 4, 0),    # 48 pixels in 64 columns: two groups of 32
    (27, 9, 9, 0),    # 243 pixels in 256 columns: one full batch
    (20, 10, 5, 2),   # 300 pixels in 320 columns: a batch and two groups, windows over the edge
    (39, 13, 13, 0),  # 507 pixels in 512 columns: two full batches
    (34, 17, 17, 0),  # 867 pixels in 896 columns: a last batch of four groups, odd rows
], ids=lambda v: str(v))
def test_window_rows_at_batch_edges(image, patch, stride, pad):
    cfg = vit_tiny(batch=3, image=image, patch=patch, patch_stride=stride, patch_pad=pad)
    w = make_weights(cfg, 57, stress=True)
    inp = make_vit_inputs(cfg, 57)
    got = run_vit(cfg, w, inp)
    assert np.isfinite(got).all()
    assert_parity(got, R.vit_encoder(cfg, w, inp), f"windows of {patch} x {patch}")
