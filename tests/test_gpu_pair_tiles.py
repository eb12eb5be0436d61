"""The kernel that multiplies pairs of 128 weight rows (csrc/tc_stream.cu, tc_pair_kernel) where its work ends: matrices of half a pair
and of one step, ragged last rows, tiles that are whole and tiles that are claimed in parts, tiles of few and of 32 activation rows."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter", [(128, 128), (384, 256), (1152, 640), (512, 12288)])
def test_fp8_projections_of_more_than_64_positions(gpu_lib, hidden, inter):
    """Dense gate (inter x hidden) and down (hidden x inter) against FP64: 1 to 96 steps, 1 to 48 pairs; 12288 rows past 300 positions
    are 480 tiles, of which most are whole. The bound is that of the same products up to 64 positions."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.hidden, c.dense_inter = 1, hidden, inter
    spec = synth.Spec(c, [0], [1], with_head=False)
    tensors = synth.make_model(spec, seed=3, recipe="spread")
    eng, _ = common.build_models(spec, tensors, 512, oracle=False, options={"allow_partial": 1})
    rng = np.random.default_rng(4)
    for name in ("mlp.gate_proj", "mlp.down_proj"):
        full = f"layers.0.{name}.weight"
        arr, _, sc = tensors[full]
        w = synth.E4M3_TABLE[arr].astype(np.float64) * np.repeat(np.repeat(sc, 128, 0), 128, 1)[:arr.shape[0], :arr.shape[1]]
        x = (rng.standard_normal((300, w.shape[1])) * np.exp2(rng.integers(-8, 9, (300, 1)))).astype(np.float32)
        for T in (65, 96, 97, 136, 300):
            got, want = eng.op_matvec(full, x[:T]), x[:T].astype(np.float64) @ w.T
            scale = np.abs(want).max(axis=1, keepdims=True) + 1e-30
            assert np.max(np.abs(got - want) / scale) < 2e-6, (name, T)
            assert np.array_equal(eng.op_matvec(full, x[:T]), got), (name, T)
    eng.close()


@pytest.mark.parametrize("hidden,inter", [(128, 128), (512, 2048), (896, 1152)])
def test_experts_whole_and_in_parts(gpu_lib, binding, hidden, inter):
    """Two tokens (every tile claimed, in one to four parts) to 300 (several hundred tiles, most of them whole); 896 rows of the down
    product end in the middle of a pair."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.n_experts, c.topk, c.moe_inter, c.hidden = 1, 4, 2, inter, hidden
    spec = synth.Spec(c, [0], [0], with_head=False)
    tensors = synth.make_model(spec, seed=8, recipe="spread")
    eng, orc = common.build_models(spec, tensors, 64, binding, options={"allow_partial": 1})
    for T in (2, 5, 33, 300):
        x = np.random.default_rng(T).standard_normal((T, c.hidden)).astype(np.float32)
        assert common.rel_err(eng.op_moe(0, x), orc.op_moe(0, x)) < 1e-5, T
        assert common.rel_err(eng.op_moe(0, x, False), orc.op_moe(0, x, False)) < 1e-5, T
    eng.close(); orc.close()
