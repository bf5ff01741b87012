"""Activations of the GEMM epilogue where they can go wrong (-m gpu): values that are not finite, large
ones, and the relative accuracy of GELU near zero."""
import dataclasses
import math

import numpy as np
import pytest

from mononn_b200 import bert_tiny, compile_encoder, make_inputs, make_weights
from oracle import ref_encoder as R
from tests.helpers import assert_parity
from tests.test_gpu_parity import run_module

pytestmark = pytest.mark.gpu


def run_with_bias(act, value):
    """One FFN-up bias set to `value`; what the device and the oracle make of it."""
    cfg = dataclasses.replace(bert_tiny(batch=2, seq=9), act=act)
    w = make_weights(cfg, 17, stress=True)
    w["layer0.ffn.up.b"][37] = value
    inp = make_inputs(cfg, 17)
    mod = compile_encoder(cfg, barrier_timeout_us=500000)
    mod.set_weights(w)
    got = run_module(mod, cfg, inp)
    mod.close()
    with np.errstate(all="ignore"):
        return got, R.bert_encoder(cfg, w, inp)


@pytest.mark.parametrize("act", ["gelu_erf", "quick_gelu", "gelu_tanh"])
@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf], ids=str)
def test_what_is_not_finite_is_passed_on(act, value):
    """f(NaN) and f(-inf) = -inf * 0 are NaN, f(inf) is inf: each reaches every column of every row through
    FFN-down and the norm behind it."""
    got, want = run_with_bias(act, value)
    assert np.isnan(want).all() and np.isnan(got).all()


@pytest.mark.parametrize("act", ["gelu_erf", "quick_gelu", "gelu_tanh"])
@pytest.mark.parametrize("value", [3e4, -3e4], ids=str)
def test_activations_of_large_values(act, value):
    got, want = run_with_bias(act, value)
    assert_parity(got, want, f"{act} of {value}")


def test_gelu_keeps_its_relative_accuracy_near_zero():
    """gelu of f16 values of standard deviation 0.05, alone: everything in front of FFN-up is zero, its bias
    holds the values, FFN-down is the identity. The output is then the norm of the stored GELU
    values. A relative error r moves a stored f16 value to its neighbour with a probability of at
    most 2^11 r: 0.1 % for GELU's 5e-7, twice, and as much again for the norm's f32 arithmetic (a GELU
    that is off by 1e-5 moves 0.8 % of them)."""
    n = 1024
    cfg = bert_tiny(batch=1, seq=2, hidden=n, ffn=n)
    w = {k: np.zeros_like(v) for k, v in make_weights(cfg, 3).items()}
    w["layer0.ffn.down.w"] = np.eye(n, dtype=np.float32)
    w["layer0.ffn.ln.gamma"] = np.ones(n, np.float32)
    inp = make_inputs(cfg, 3)
    mod = compile_encoder(cfg, barrier_timeout_us=500000)
    mod.set_weights(w)
    rng = np.random.default_rng(5)
    moved = total = 0
    for _ in range(16):
        v = rng.normal(0.0, 0.05, n).astype(np.float16)
        mod.set_constant("layer0.ffn.up.b", v)
        got = run_module(mod, cfg, inp)[0].astype(np.float16)
        erf = np.array([math.erf(x / math.sqrt(2.0)) for x in v.astype(np.float64)])
        h = (0.5 * v.astype(np.float64) * (1.0 + erf)).astype(np.float16).astype(np.float64)
        want = ((h - h.mean()) / np.sqrt(h.var() + cfg.eps)).astype(np.float16)
        assert np.abs(got.astype(np.float64) - want).max() <= 4e-3  # two spacings of f16 values up to 4
        moved += int((got != want).sum())
        total += n
    mod.close()
    assert moved <= 0.003 * total, f"{moved} of {total} values off"
