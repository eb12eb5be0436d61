"""A few queries at many positions (csrc/mla.cu): the attention core's stretches summed by the CTAs that take a head's value rows, and
the selection's digits counted with and without the warp's help."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v_head,heads", [(64, 16), (256, 32), (136, 16), (36, 16)])
def test_few_queries_over_many_stretches(gpu_lib, binding, v_head, heads):
    """Value rows that fill a CTA's 128, that end within a warp's eight, and a second CTA with eight of them; one to four queries (four take
    the tiles); few stretches (48 positions each) and many; with and without a selection."""
    c = pkg.Config(hidden=512, n_layers=1, vocab=64, rms_eps=1e-5, hc_mult=4, hc_iters=20, hc_eps=1e-6, kda_heads=4, kda_head_dim=64, conv_k=4,
                   gate_lb=-5.0, mla_heads=heads, q_lora=192, kv_lora=512, qk_nope=64, v_head=v_head, index_topk=640, index_kpool=4, index_heads=8,
                   index_dim=48, n_experts=22, topk=2, n_shared=1, moe_inter=128, dense_inter=256, routed_scale=2.5, norm_topk=1, swiglu_limit=10.0,
                   fp8_block_r=128, fp8_block_c=128)
    spec = synth.Spec(c, [1], [0], with_head=False, only="mla")
    cap = 1600
    eng, orc = common.build_models(spec, synth.make_model(spec, seed=31, recipe="spread"), cap, binding, options={"allow_partial": 1, "latent_bf16": 1})
    rng = np.random.default_rng(6)
    lat = synth.bf16_round(rng.standard_normal((cap, c.kv_lora)).astype(np.float32))
    idx = rng.standard_normal(2 * cap * c.index_dim + (cap // c.index_kpool) * c.index_dim).astype(np.float32)
    for m in (eng, orc):
        m.state_write(0, 1, 0, lat)
        m.state_write(0, 2, 0, idx)
    for cached, T in ((60, 1), (62, 3), (500, 2), (1500, 1), (1502, 3), (1506, 4)):
        x = rng.standard_normal((T, c.hidden)).astype(np.float32)
        (g, gs), (w, ws) = eng.op_mla(0, x, cached), orc.op_mla(0, x, cached)
        assert (gs is None) == (ws is None) and (gs is None or np.array_equal(gs, ws)), (cached, T)
        # the new positions' latents are rounded to BF16 here: 2^-9 of a latent at most, whatever its weight
        assert common.rel_err(g, w) < 2.0 ** -9, (cached, T)
    eng.close(); orc.close()
