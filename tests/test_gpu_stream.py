"""The tensor-core streaming kernels (csrc/tc_stream.cu) at the sizes where their tiles end: rows of W that do
not fill a 128-row tile, columns that do not fill a unit (256 FP8 / 128 BF16), 2..64 positions around the multiples
of 8 and the step from one to two groups of 32 rows, matrices of one unit, and experts with few and with many rows."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter", [(128, 128), (384, 256), (1152, 640)])
def test_projections_at_the_edges_of_tiles(gpu_lib, hidden, inter):
    """Dense gate (inter x hidden) and down (hidden x inter) in FP8, b_proj (few rows) and o_proj in BF16, against FP64."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.hidden, c.dense_inter, c.kda_heads = 1, hidden, inter, 3
    spec = synth.Spec(c, [0], [1], with_head=False)
    tensors = synth.make_model(spec, seed=3, recipe="spread")
    eng, _ = common.build_models(spec, tensors, 64, oracle=False, options={"allow_partial": 1})
    rng = np.random.default_rng(4)
    for name in ("mlp.gate_proj", "mlp.down_proj", "self_attn.q_proj", "self_attn.b_proj", "self_attn.o_proj"):
        full = f"layers.0.{name}.weight"
        arr, dt, sc = tensors[full]
        if dt == pkg.DT_FP8:
            w = synth.E4M3_TABLE[arr].astype(np.float64) * np.repeat(np.repeat(sc, 128, 0), 128, 1)[:arr.shape[0], :arr.shape[1]]
        else:
            w = (arr.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
        x = (rng.standard_normal((64, w.shape[1])) * np.exp2(rng.integers(-8, 9, (64, 1)))).astype(np.float32)
        for T in (2, 7, 8, 9, 31, 32, 33, 40, 63, 64):
            got, want = eng.op_matvec(full, x[:T]), x[:T].astype(np.float64) @ w.T
            scale = np.abs(want).max(axis=1, keepdims=True) + 1e-30
            assert np.max(np.abs(got - want) / scale) < 2e-6, (name, T)
    eng.close()


@pytest.mark.parametrize("T", [2, 9, 31, 33, 64, 65, 300])
def test_experts_with_few_and_with_many_rows(gpu_lib, binding, T):
    """Four experts of which every token takes two and the shared one: slots of up to T rows, cut into tiles of 32."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.n_experts, c.topk, c.moe_inter, c.hidden = 1, 4, 2, 384, 256
    spec = synth.Spec(c, [0], [0], with_head=False)
    tensors = synth.make_model(spec, seed=8, recipe="spread")
    eng, orc = common.build_models(spec, tensors, 64, binding, options={"allow_partial": 1})
    x = np.random.default_rng(T).standard_normal((T, c.hidden)).astype(np.float32)
    assert common.rel_err(eng.op_moe(0, x), orc.op_moe(0, x)) < 1e-5
    assert common.rel_err(eng.op_moe(0, x, False), orc.op_moe(0, x, False)) < 1e-5
    eng.close(); orc.close()


def test_prompt_of_several_attention_chunks(gpu_lib, binding):
    """A prompt longer than the 64 positions of the attention core and the router, then decode steps on its state."""
    spec = synth.tiny_spec()
    tensors = synth.make_model(spec, seed=31, recipe="spread")
    eng, orc = common.build_models(spec, tensors, 300, binding)
    ids = np.random.default_rng(6).integers(0, spec.cfg.vocab, 270).astype(np.int32)
    g, w = eng.forward(ids)[0], orc.forward(ids)[0]
    for tok in (3, 77):
        assert common.rel_err(g, w) < 1e-3 and int(g.argmax()) == int(w.argmax())
        g, w = eng.forward([tok])[0], orc.forward([tok])[0]
    eng.close(); orc.close()


@pytest.mark.parametrize("hidden", [512, 4096])
def test_stream_mixing_of_many_positions(gpu_lib, binding, hidden):
    """More positions than clusters that fit the GPU at once: one CTA per position; the second layer also applies what the
    first one owes to the streams. Few pieces per thread and many."""
    c = pkg.Config(hidden=hidden, n_layers=2, vocab=64, rms_eps=1e-5, hc_mult=4, hc_iters=20, hc_eps=1e-6,
                   kda_heads=4, kda_head_dim=64, conv_k=4, gate_lb=-5.0, mla_heads=4, q_lora=192, kv_lora=128,
                   qk_nope=64, v_head=64, index_topk=16, index_kpool=4, index_heads=4, index_dim=32,
                   n_experts=40, topk=2, n_shared=1, moe_inter=128, dense_inter=256, routed_scale=2.5,
                   norm_topk=1, swiglu_limit=10.0, fp8_block_r=128, fp8_block_c=128)
    spec = synth.Spec(c, [0, 1], [1, 0], with_head=True)
    tensors = synth.make_model(spec, seed=23, recipe="spread")
    eng, orc = common.build_models(spec, tensors, 128, binding)
    ids = np.random.default_rng(6).integers(0, c.vocab, 85).astype(np.int32)
    assert common.rel_err(eng.forward(ids)[0], orc.forward(ids)[0]) < 1e-4
    eng.close(); orc.close()


@pytest.mark.parametrize("T", [16, 17, 32, 33, 64, 65, 150])
def test_router_of_many_tokens(gpu_lib, binding, T):
    """Tiles of 32 tokens x 32 experts with ragged edges of both, columns in one and in several stretches."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.n_experts, c.topk, c.hidden = 1, 45, 4, 384
    spec = synth.Spec(c, [0], [0], with_head=False)
    tensors = synth.make_model(spec, seed=9, recipe="spread")
    eng, orc = common.build_models(spec, tensors, 64, binding, options={"allow_partial": 1})
    x = np.random.default_rng(T).standard_normal((T, c.hidden)).astype(np.float32)
    assert common.rel_err(eng.op_moe(0, x), orc.op_moe(0, x)) < 1e-5
    gi, gw = eng.last_picks((T - 1) % 64 + 1)
    wi, ww = orc.op_router(0, x)
    assert np.array_equal(gi, wi[-len(gi):]) and common.rel_err(gw, ww[-len(gi):]) < 1e-6
    eng.close(); orc.close()


def _moe_engine(hidden, inter, cap, rank=0, ranks=1):
    c = synth.layer_spec("moe", n_experts=24).cfg.copy()
    c.hidden, c.moe_inter, c.topk = hidden, inter, 4
    spec = synth.Spec(c, [0], [0], with_head=False)
    eng = pkg.Engine(c, spec.is_mla, spec.is_dense, cap, 0, rank, ranks)
    eng.set_option("allow_partial", 1)
    eng.load_all(synth.moe_layer_trunk(spec, 5))
    for x in range(rank * c.n_experts // ranks, (rank + 1) * c.n_experts // ranks):
        eng.fill_expert(0, x, 5, *synth.expert_scales(c, 0, x, 5))
    eng.finalize()
    return spec, eng


@pytest.mark.parametrize("hidden,inter", [(4096, 2048), (2304, 1152)])
def test_expert_rows_do_not_depend_on_what_is_beside_them(gpu_lib, hidden, inter):
    """Sixteen, eight, nine and five units to a tile, cut between the CTAs at other places in every launch below: a row of an
    expert has the same bits in any batch, on every rank of a group and on one GPU, and in every run."""
    spec, one = _moe_engine(hidden, inter, 512)
    ranks = [_moe_engine(hidden, inter, 64, r, 2)[1] for r in (0, 1)]
    x = np.random.default_rng(7).standard_normal((300, hidden)).astype(np.float32)
    picks, shared = one.debug_moe_rows(0, x)
    for first, n in ((0, 2), (3, 7), (20, 31), (200, 64)):
        rows = slice(first, first + n)
        p, s = one.debug_moe_rows(0, x[rows])
        assert np.array_equal(p, picks[rows]) and np.array_equal(s, shared[rows]), n
        parts = [e.debug_moe_rows(0, x[rows]) for e in ranks]
        for r, (p, s) in enumerate(parts):
            assert np.array_equal(s, shared[rows]), (n, r)
        assert not np.any((parts[0][0] != 0) & (parts[1][0] != 0))
        assert np.array_equal(parts[0][0] + parts[1][0], picks[rows]), n
    for n in (64, 300):
        first = one.op_moe(0, x[:n])
        for _ in range(3):
            assert np.array_equal(one.op_moe(0, x[:n]), first), n
    for e in (one, *ranks):
        e.close()


def test_profile_tells_the_expert_phases_of_a_batch_apart(gpu_lib):
    """Option "profile": router and plan, gate/up, down and combine each take measurable time; gate/up is two of the three matrices."""
    import ctypes as C
    spec, eng = _moe_engine(2048, 1024, 64)
    x = np.random.default_rng(3).standard_normal((48, 2048)).astype(np.float32)
    eng.op_moe(0, x)
    ms, count = (C.c_float * 8)(), C.c_long(0)
    read = eng.L.g5b_engine_profile_read
    read.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int]
    eng.set_option("profile", 1)
    for _ in range(20):
        eng.op_moe(0, x)
    assert read(eng.handle, C.addressof(ms), 8, C.addressof(count), 1) == 0 and count.value == 20
    router, gateup, down, combine = (v / 20 for v in list(ms)[:4])
    # an empty phase is the 1 to 2 us between two events; these are launches of tens of microseconds
    assert min(router, gateup, down) > 5e-3 and combine > 1e-3, list(ms)
    assert down < gateup, list(ms)
    eng.close()


def test_prompts_and_batches_repeat_bit_for_bit(gpu_lib):
    """The same prompt and the same step of a batch of sequences again, from the same state: the same logits."""
    spec = synth.tiny_spec()
    tensors = synth.make_model(spec, seed=33, recipe="spread")
    eng, _ = common.build_models(spec, tensors, 300, oracle=False, options={"sequences": 9})
    rng = np.random.default_rng(8)
    ids, step = rng.integers(0, spec.cfg.vocab, 270).astype(np.int32), rng.integers(0, spec.cfg.vocab, 9).astype(np.int32)

    def both():
        eng.use_sequence(0)
        eng.reset()
        prompt = eng.forward(ids)[0]
        eng.reset()
        eng.synth_session(4, 100)
        return prompt, eng.decode_batch(step)[0]

    first = both()
    for _ in range(3):
        again = both()
        assert np.array_equal(again[0], first[0]) and np.array_equal(again[1], first[1])
    eng.close()
