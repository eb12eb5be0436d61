"""One position of each of several sequences (csrc/kda.cu, kda_each_kernel): both head sizes, states that differ from sequence to
sequence, several steps, against separate sessions of the CPU path."""
import numpy as np
import pytest

import common
import synth

pkg = synth.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim,heads,conv", [(128, 3, 4), (64, 5, 4), (128, 2, 3)])
def test_batched_kda_steps_match_separate_sessions(gpu_lib, binding, head_dim, heads, conv):
    """A width of 3 takes the kernels for several positions."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.kda_head_dim, c.kda_heads, c.conv_k = 2, head_dim, heads, conv
    spec = synth.Spec(c, [0, 0], [1, 1], with_head=True)
    tensors = synth.make_model(spec, seed=11, recipe="spread")
    S, rng = 3, np.random.default_rng(2)
    eng, _ = common.build_models(spec, tensors, 32, oracle=False, options={"sequences": S})
    sessions = []
    for q in range(S):
        orc = common.build_models(spec, tensors, 32, binding, engine=False)[1]
        ids = rng.integers(0, c.vocab, 5).astype(np.int32)
        eng.use_sequence(q)
        assert common.rel_err(eng.forward(ids)[0], orc.forward(ids)[0]) < 1e-4
        sessions.append(orc)
    for _ in range(4):
        ids = rng.integers(0, c.vocab, S).astype(np.int32)
        got = eng.decode_batch(ids)[0]
        for q, orc in enumerate(sessions):
            assert common.rel_err(got[q], orc.forward(ids[q:q + 1])[0]) < 1e-4, q
    eng.close()
    for orc in sessions:
        orc.close()
