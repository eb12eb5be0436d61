"""The kernels that multiply with the FP64 matrix instruction (csrc/f64_tile.cuh, mhc.cu, mla.cu) at the sizes where their tiles
end: 8, 16, 32 and 64 rows, 64 columns, stretches of positions and of router columns, eight positions of a mixing site."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu


def _config(**kw):
    return pkg.Config(**{**dict(hidden=512, n_layers=2, vocab=64, rms_eps=1e-5, hc_mult=4, hc_iters=20, hc_eps=1e-6,
                                kda_heads=4, kda_head_dim=64, conv_k=4, gate_lb=-5.0, mla_heads=64, q_lora=192, kv_lora=128,
                                qk_nope=64, v_head=64, index_topk=64, index_kpool=4, index_heads=8, index_dim=48,
                                n_experts=22, topk=2, n_shared=1, moe_inter=128, dense_inter=256, routed_scale=2.5,
                                norm_topk=1, swiglu_limit=10.0, fp8_block_r=128, fp8_block_c=128), **kw})


@pytest.mark.parametrize("hidden,T", [(512, 16), (512, 17), (640, 23), (512, 24), (640, 70), (4096, 31)])
def test_mixing_sites_in_groups_of_eight(gpu_lib, binding, hidden, T):
    """Whole and ragged groups of eight; 64, 80 and 512 columns per CTA; with and without a pending stream expansion."""
    c = _config(hidden=hidden)
    spec = synth.Spec(c, [0, 0], [1, 1], with_head=True)
    eng, orc = common.build_models(spec, synth.make_model(spec, seed=23, recipe="spread"), 128, binding)
    h = np.random.default_rng(T).standard_normal((T, c.hc_mult, hidden)).astype(np.float32)
    # FP32 products of the layers around the sites: the bound of every layer test here
    assert common.rel_err(eng.op_decoder_layer(0, h, 0), orc.op_decoder_layer(0, h, 0)) < 1e-5
    eng.close(); orc.close()


@pytest.mark.parametrize("T", [1, 16])
def test_mixing_sites_with_extreme_mixer_elements(gpu_lib, binding, T):
    """Infinite elements (no place among the scaled ones), the smallest subnormal, zeros and the largest finite one, one position
    and groups of eight: what the CPU path's FP64 sums give."""
    c = _config()
    spec = synth.Spec(c, [0, 0], [1, 1], with_head=True)
    tensors = synth.make_model(spec, seed=23, recipe="spread")
    h = np.abs(np.random.default_rng(4).standard_normal((T, 4, c.hidden))).astype(np.float32)
    for values in ((0x0001, 0x8001, 0x0000, 0x8000, 0x0080), (0x3000, 0x7f7f, 0x0001, 0xb000, 0x0000), (0x7f80, 0x0001, 0x3f80, 0x0000, 0x3f80)):
        arr, dt, sc = tensors["layers.0.hc_attn_fn"]
        arr = arr.copy()
        arr[1, :len(values)] = values                       # a row of the collapse's gates
        eng, orc = common.build_models(spec, {**tensors, "layers.0.hc_attn_fn": (arr, dt, sc)}, 16, binding)
        g, w = eng.op_decoder_layer(0, h, 0), orc.op_decoder_layer(0, h, 0)
        assert np.isfinite(w).all() and common.rel_err(g, w) < 1e-5, values
        eng.close(); orc.close()


@pytest.mark.parametrize("n_experts", [22, 23, 288])
def test_router_of_several_tokens(gpu_lib, binding, n_experts):
    """Ragged tiles of experts, an odd number of them (the untiled path), stretches of the columns; indices identical."""
    c = _config(n_experts=n_experts, hidden=1152)
    spec = synth.Spec(c, [0, 0], [0, 0], with_head=True)
    eng, orc = common.build_models(spec, synth.make_model(spec, seed=5, recipe="spread"), 16, binding)
    rng = np.random.default_rng(n_experts)
    for T in (16, 17, 32, 33, 64, 65, 130):
        x = rng.standard_normal((T, c.hidden)).astype(np.float32)
        eng.op_moe(0, x)                                    # (the router op itself takes the untiled path)
        (gi, gw), (wi, ww) = eng.last_picks((T - 1) % 64 + 1), orc.op_router(0, x)
        assert np.array_equal(gi, wi[-len(gi):]) and common.rel_err(gw, ww[-len(gi):]) < 1e-6, T
    eng.close(); orc.close()


@pytest.mark.parametrize("index_heads,kv_lora,latent_bf16", [(8, 128, 0), (32, 512, 0), (12, 128, 0), (16, 512, 1)])
def test_attention_of_several_queries(gpu_lib, binding, index_heads, kv_lora, latent_bf16):
    """Absorption, FP64 attention core and pool scores: everything visible, a selection, more than one stretch of 512 visible positions;
    12 indexer heads take the untiled scores. Selections identical."""
    c = _config(n_layers=1, index_heads=index_heads, kv_lora=kv_lora, qk_nope=96, index_topk=640)
    spec = synth.Spec(c, [1], [0], with_head=False, only="mla")
    cap = 1024
    eng, orc = common.build_models(spec, synth.make_model(spec, seed=6, recipe="spread"), cap, binding, options={"allow_partial": 1, "latent_bf16": latent_bf16})
    rng = np.random.default_rng(index_heads)
    lat = synth.bf16_round(rng.standard_normal((cap, kv_lora)).astype(np.float32))
    idx = rng.standard_normal(2 * cap * c.index_dim + (cap // c.index_kpool) * c.index_dim).astype(np.float32)
    for m in (eng, orc):
        m.state_write(0, 1, 0, lat)
        m.state_write(0, 2, 0, idx)
    for T, cached in ((2, 0), (7, 500), (8, 0), (9, 505), (16, 630), (17, 800), (33, 470), (65, 610), (70, 0)):
        x = synth.bf16_round(rng.standard_normal((T, c.hidden)).astype(np.float32))
        (g, gs), (w, ws) = eng.op_mla(0, x, cached), orc.op_mla(0, x, cached)
        assert (gs is None) == (ws is None) and (gs is None or np.array_equal(gs, ws)), (T, cached)
        assert common.rel_err(g, w) < (3e-3 if latent_bf16 else 2e-5), (T, cached)
    eng.close(); orc.close()
