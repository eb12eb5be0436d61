"""The tensor-core attention core (csrc/mla.cu, mla_flash_kernel) where a CTA walks several chunks of 48 positions: what the
additions of the chunks' sums may lose, references that rise from chunk to chunk, a second group of 512 queries, selections. Against
FP64 sums and against the FP64 core on the same cache."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu
HEADS, V, KL, HIDDEN = 64, 16, 512, 1024


def _layer(index_topk, cap, **changed):
    """Output column c is latent column c % 512 of head c / 16's sum: the value rows and the output projection pick, exactly."""
    c = pkg.Config(hidden=HIDDEN, n_layers=1, vocab=64, rms_eps=1e-5, hc_mult=4, hc_iters=20, hc_eps=1e-6, kda_heads=4, kda_head_dim=64, conv_k=4,
                   gate_lb=-5.0, mla_heads=HEADS, q_lora=192, kv_lora=KL, qk_nope=64, v_head=V, index_topk=index_topk, index_kpool=4, index_heads=8,
                   index_dim=48, n_experts=22, topk=2, n_shared=1, moe_inter=128, dense_inter=256, routed_scale=2.5, norm_topk=1, swiglu_limit=10.0,
                   fp8_block_r=128, fp8_block_c=128)
    spec = synth.Spec(c, [1], [0], with_head=False, only="mla")
    tensors = synth.make_model(spec, seed=41, recipe="spread")
    p = "layers.0.self_attn."
    kv_b = np.zeros((HEADS, 64 + V, KL), np.float32)
    kv_b[:, :64, :64] = np.eye(64)                            # a query's scores come from the first 64 columns
    for h in range(HEADS):
        kv_b[h, 64 + np.arange(V), (h * V + np.arange(V)) % KL] = 1.0
    tensors[p + "kv_b_proj.weight"] = (synth.to_bf16_bits(kv_b.reshape(-1, KL)), pkg.DT_BF16, None)
    tensors[p + "o_proj.weight"] = (synth.to_bf16_bits(np.eye(HIDDEN, dtype=np.float32)), pkg.DT_BF16, None)
    for name, value in changed.items():
        t = tensors[p + name + ".weight"]
        tensors[p + name + ".weight"] = (np.full_like(t[0], value), t[1], t[2])
    return common.build_models(spec, tensors, cap, oracle=False, options={"allow_partial": 1, "latent_bf16": 1})[0], c


@pytest.mark.parametrize("T", [64, 150])
def test_small_chunks_behind_a_large_one(gpu_lib, T):
    """Every position weighs the same. The first has 256 in a column, the others 2^-22 to 1.25 times that: 48 of them are less than half of
    the sum's last place, 2^-15, so an FP32 sum over the chunks stays at 256 and loses 1800 of them, 2e-6 of it. In a CTA that takes all
    of a query's chunks only the first one's own small values may go (2^-24), and the result's rounding (2^-24); where a query is cut
    into stretches each ends in a float (a third 2^-24)."""
    cached, cap = 1900, 2304
    eng, c = _layer(2048, cap, q_b_proj=0)
    rng = np.random.default_rng(8)
    lat = np.zeros((cap, KL), np.float32)
    lat[:cached] = synth.bf16_round((rng.uniform(1.0, 1.25, (cached, KL)) * 2.0 ** -22).astype(np.float32))
    lat[0] = 256.0
    eng.state_write(0, 1, 0, lat)
    got, sel = eng.op_mla(0, np.zeros((T, HIDDEN), np.float32), cached)      # the new positions' latents are zero
    assert sel is None
    want = np.tile(lat.astype(np.float64).sum(axis=0), HIDDEN // KL)[None] / (cached + 1.0 + np.arange(T))[:, None]
    assert common.rel_err(got, want) < 3 * 2.0 ** -24
    eng.close()


@pytest.mark.parametrize("rising", [0, 1])
@pytest.mark.parametrize("index_topk,cached,T", [(2048, 1400, 150), (2048, 1400, 600), (640, 1400, 530), (640, 1400, 64), (2048, 1400, 5)])
def test_several_chunks_match_the_fp64_core(gpu_lib, index_topk, cached, T, rising):
    """Ordinary scores, below 4 in size, and scores that grow by 0 to 14 a chunk up to 60, where the largest of a later chunk is far above, a little
    above and below 16 more than what came before. A score's four products of 16 columns are cut off at its last place each (2^-22, 2^-18), the
    FP64 core rounds it to a float (half of that), and an error there is a relative one of a weight: 4.5 places, 1.1e-6 and
    1.7e-5. On top of that three products of a chunk's weighted sum, 1.2e-7 each."""
    cap = 2304
    eng, c = _layer(index_topk, cap)
    rng = np.random.default_rng(9)
    lat = rng.standard_normal((cap, KL)).astype(np.float32)
    if rising:
        lat[:, :64] = (np.minimum(7 * (np.arange(cap) // 48), 28) + rng.uniform(0, 1, cap))[:, None] * rng.standard_normal(64)[None]
    idx = rng.standard_normal(2 * cap * c.index_dim + (cap // c.index_kpool) * c.index_dim).astype(np.float32)
    eng.state_write(0, 1, 0, synth.bf16_round(lat))
    eng.state_write(0, 2, 0, idx)
    x = rng.standard_normal((T, HIDDEN)).astype(np.float32)
    got, sel = eng.op_mla(0, x, cached)
    eng.set_option("mla_tensor", 0)
    want, sel64 = eng.op_mla(0, x, cached)
    eng.set_option("mla_tensor", 1)
    assert (sel is None) == (index_topk == 2048) and (sel is None or np.array_equal(sel, sel64))
    assert np.isfinite(got).all()
    assert common.rel_err(got, want) < (2e-5 if rising else 2e-6)
    eng.close()


@pytest.mark.parametrize("index_topk,T,taken", [(3064, 1, True), (3080, 1, True), (3080, 64, True), (4092, 1, True), (4092, 5, True), (4096, 1, False)])
def test_as_many_positions_as_the_core_takes(gpu_lib, index_topk, T, taken):
    """Up to 4096 positions a query, 86 chunks and more than the second kernel has places for stretches; beyond, the FP64 core
    (the same bits with and without the option). Scores below 4: the bound of the test above."""
    cap, cached = 4608, 4500
    eng, c = _layer(index_topk, cap)
    rng = np.random.default_rng(10)
    eng.state_write(0, 1, 0, synth.bf16_round(rng.standard_normal((cap, KL)).astype(np.float32)))
    eng.state_write(0, 2, 0, rng.standard_normal(2 * cap * c.index_dim + (cap // c.index_kpool) * c.index_dim).astype(np.float32))
    x = rng.standard_normal((T, HIDDEN)).astype(np.float32)
    got, sel = eng.op_mla(0, x, cached)
    eng.set_option("mla_tensor", 0)
    want, sel64 = eng.op_mla(0, x, cached)
    assert np.array_equal(sel, sel64) and len(sel) >= index_topk
    assert np.array_equal(got, want) != taken
    assert common.rel_err(got, want) < 2e-6
    eng.close()
