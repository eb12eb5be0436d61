"""The router's selection for two and more tokens (csrc/moe.cu, router_select_kernel), as the layer runs it: picks and their order with
equal scores, with experts that cannot be selected, and at the sizes of its tiles of eight tokens."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu
GATE, BIAS = "layers.0.mlp.gate.weight", "layers.0.mlp.gate.e_score_correction_bias"


def _models(binding, n_experts, topk, change):
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.n_experts, c.topk, c.moe_inter, c.hidden = 1, n_experts, topk, 128, 384
    spec = synth.Spec(c, [0], [0], with_head=False)
    tensors = synth.make_model(spec, seed=15, recipe="spread")
    (gate, gdt, gs), (bias, bdt, bs) = tensors[GATE], tensors[BIAS]
    gate, bias = gate.copy(), bias.copy()
    change(gate, bias)
    tensors[GATE], tensors[BIAS] = (gate, gdt, gs), (bias, bdt, bs)
    return *common.build_models(spec, tensors, 64, binding, options={"allow_partial": 1}), c


def _compare(eng, orc, c, tokens):
    for T in tokens:
        x = np.random.default_rng(T).standard_normal((T, c.hidden)).astype(np.float32)
        eng.op_moe(0, x)
        (gi, gw), (wi, ww) = eng.last_picks(T), orc.op_router(0, x)
        assert np.array_equal(gi, wi), T
        assert common.rel_err(gw, ww) < 1e-6, T
    eng.close(); orc.close()
    return gi


@pytest.mark.parametrize("n_experts,topk", [(32, 5), (64, 7), (70, 8), (288, 8), (288, 15)])
def test_equal_scores(gpu_lib, binding, n_experts, topk):
    """Experts 2i + 1 and 2i + 2 share their row and bias: pairs lie within a warp and across two (31 and 32), and an odd number
    of picks cuts one. The lower expert goes first."""
    def change(gate, bias):
        gate[2::2], bias[2::2] = gate[1:-1:2], bias[1:-1:2]
        bias[1:-1] += 1.0                                    # (the pairs before expert 0 and the last one)
    eng, orc, c = _models(binding, n_experts, topk, change)
    picks = _compare(eng, orc, c, (2, 3, 4, 7, 8, 9, 15, 16, 33))
    cut = picks[:, topk - 1] if topk % 2 else picks[:, topk - 2]
    assert (cut % 2 == 1).all() and (picks[:, 0] % 2 == 1).all() and (picks[:, 1] == picks[:, 0] + 1).all()


def test_all_scores_equal(gpu_lib, binding):
    def change(gate, bias):
        gate[:] = gate[0]
        bias[:] = bias[0]
    eng, orc, c = _models(binding, 96, 8, change)
    assert (_compare(eng, orc, c, (2, 6, 13)) == np.arange(8)).all()


@pytest.mark.parametrize("left", [8, 9, 40])
def test_experts_that_cannot_be_selected(gpu_lib, binding, left):
    """A bias of -inf or NaN takes an expert out; as many as a token picks are left, or a few more."""
    def change(gate, bias):
        out = np.random.default_rng(left).permutation(len(bias))[left:]
        bias[out[::2]], bias[out[1::2]] = -np.inf, np.nan
    eng, orc, c = _models(binding, 96, 8, change)
    _compare(eng, orc, c, (2, 5, 8, 11, 40))
