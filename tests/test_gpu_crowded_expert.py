"""Experts with more rows than the call has tokens (csrc/tc_stream.cu, tc_pair_kernel): places that nothing selectable is left for all go
to expert 0, so a few rows of NaN, or a bias that leaves fewer experts than a token picks, give it several rows per token."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu
GATE, BIAS = "layers.0.mlp.gate.weight", "layers.0.mlp.gate.e_score_correction_bias"


def _layer(binding=None, bias=None):
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.n_experts, c.topk, c.moe_inter, c.hidden = 1, 24, 8, 256, 512
    spec = synth.Spec(c, [0], [0], with_head=False)
    tensors = synth.make_model(spec, seed=14, recipe="spread")
    if bias is not None:
        arr, dt, sc = tensors[BIAS]
        tensors[BIAS] = (bias.astype(arr.dtype), dt, sc)
    return common.build_models(spec, tensors, 64, binding, oracle=binding is not None, options={"allow_partial": 1}), c


@pytest.mark.parametrize("T", [2, 3, 5, 8, 9, 12, 17, 24, 31, 40])
def test_rows_of_nan_beside_ordinary_ones(gpu_lib, binding, T):
    """All rows but two (one of two) are NaN: eight rows of expert 0 each. The others are what the CPU path gives them alone."""
    (eng, orc), c = _layer(binding)
    x = np.full((T, c.hidden), np.nan, np.float32)
    some = [T - 1] if T == 2 else [1, T - 1]
    x[some] = np.random.default_rng(T).standard_normal((len(some), c.hidden)).astype(np.float32)
    got = eng.op_moe(0, x)
    assert common.rel_err(got[some], orc.op_moe(0, x[some])) < 1e-5
    assert np.isnan(np.delete(got, some, axis=0)).all()
    ordinary = np.random.default_rng(1).standard_normal((T, c.hidden)).astype(np.float32)
    assert common.rel_err(eng.op_moe(0, ordinary), orc.op_moe(0, ordinary)) < 1e-5      # (and nothing is left behind)
    eng.close(); orc.close()


@pytest.mark.parametrize("T", [2, 7, 16, 19, 33])
def test_fewer_experts_than_picks(gpu_lib, T):
    """Three experts can be selected, five of a token's eight places go to expert 0: the same picks as the untiled selection, the
    same rows as the kernels without tensor cores."""
    bias = np.full(24, -np.inf)
    bias[[5, 11, 17]] = 0.0
    (eng, _), c = _layer(bias=bias)
    x = np.random.default_rng(T).standard_normal((T, c.hidden)).astype(np.float32)
    got = eng.op_moe(0, x)
    picks, w = eng.last_picks(T)
    idx, want_w = eng.op_router(0, x)
    assert np.array_equal(picks, idx) and (idx[:, 3:] == 0).all() and common.rel_err(w, want_w) < 1e-6
    eng.set_option("expert_path", 0)
    assert common.rel_err(got, eng.op_moe(0, x)) < 1e-5
    eng.close()
