"""GEMM epilogues whose last group of 32 columns is half a group (-m gpu): tiles 16, 48, 80 and 240 columns
wide, stored as f16 (bias, GELU), transposed, and added to f32 rows (bias, split K or not)."""
import json

import pytest

from mononn_b200 import bert_tiny, compile_hlo, make_inputs, make_vit_inputs, make_weights, vit_tiny
from mononn_b200.hlo_builder import bert_hlo, vit_hlo
from mononn_b200.module import describe
from oracle import ref_encoder as R
from tests.helpers import assert_parity

pytestmark = pytest.mark.gpu

OUT_F16, OUT_F16_T, OUT_F32_RED = 0, 1, 2


def compile_with_tiles(text, names, weights, tile, split, tmp_path):
    """The module with every GEMM in tiles of `tile` columns; the output modes of its GEMMs."""
    spec = describe("hlo", text)["spec"]
    spec.update(qkv_fusion="off", row_fusion="off", out_fusion="off")
    spec.pop("gemm_spec_list")
    spec = describe("hlo", text, spec=spec)["spec"]
    for gemm in spec["gemm_spec_list"].values():
        cfg, blocks = gemm["sm100_config"], gemm["problem"]["k"] // 64
        cfg["mma_n"] = tile
        cfg["k_split"] = blocks if split and cfg["k_split"] > 1 else 1
    (tmp_path / "cluster_0").mkdir()
    (tmp_path / "cluster_0" / "best_tuning_spec.json").write_text(json.dumps(spec))
    mod = compile_hlo(text, spec_dir=str(tmp_path), barrier_timeout_us=500000)
    gemms = [o for s in mod.plan()["stages"] for o in s["ops"] if o["kind"] == "gemm"]
    assert all(o["n_tile"] == tile for o in gemms)
    mod.set_weights({names[k]: v for k, v in weights.items()})
    return mod, {o["out_mode"] for o in gemms}


@pytest.mark.parametrize("tile, split", [(16, True), (48, True), (48, False), (80, True), (240, False)])
def test_half_groups_of_a_post_norm_layer(tile, split, tmp_path):
    """Rows that end inside a tile (136 rows), biases on every GEMM, values transposed."""
    cfg = bert_tiny(batch=4, seq=34, layers=1, hidden=192, ffn=320)
    w, inp = make_weights(cfg, 95, stress=True), make_inputs(cfg, 95)
    mod, modes = compile_with_tiles(*bert_hlo(cfg), w, tile, split, tmp_path)
    assert {OUT_F16, OUT_F16_T, OUT_F32_RED} <= modes
    out = mod.run([inp["input_ids"], inp["attention_mask"], inp["token_type_ids"]])[0]
    mod.close()
    got = out[: cfg.tokens * cfg.hidden].reshape(cfg.tokens, cfg.hidden)
    assert_parity(got, R.bert_encoder(cfg, w, inp), f"tiles of {tile}")


@pytest.mark.parametrize("tile, split", [(16, True), (48, False), (80, True), (240, False)])
def test_half_groups_added_to_a_residual_stream(tile, split, tmp_path):
    cfg = vit_tiny(batch=8, image=64, layers=1, hidden=192)
    w, inp = make_weights(cfg, 96, stress=True), make_vit_inputs(cfg, 96)
    mod, modes = compile_with_tiles(*vit_hlo(cfg), w, tile, split, tmp_path)
    assert {OUT_F16, OUT_F32_RED} <= modes
    out = mod.run([inp["pixel_values"]])[0]
    mod.close()
    got = out[: cfg.tokens * cfg.hidden].reshape(cfg.tokens, cfg.hidden)
    assert_parity(got, R.vit_encoder(cfg, w, inp), f"tiles of {tile}")
