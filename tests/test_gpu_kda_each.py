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


def _small_parts_kept(step, H, D):
    """A step of sequences with the same token is one linear map of a state's columns, S -> aS - k beta u with u the sum of w_i S_i (v = 0). The
    identity as a state shows a and w. Then a column with a large value in the first of a thread's 32 rows, and the same with 0.45 of the sum's
    last place in all others: the share of these that u has kept, per head."""
    one = np.tile(np.eye(D), (H, 1, 1))
    m = step(one, one)[0]                                    # m[h][i][j] = (i == j) a_j - k_i beta w_j
    a, b, grew, known = np.zeros((H, D, D)), np.zeros((H, D, D)), np.zeros((H, D)), []
    for h in range(H):
        off = m[h] - np.diag(np.diag(m[h]))
        i0, i1 = np.argsort(-np.abs(off).max(axis=1))[:2]
        j = next(n for n in np.argsort(-np.abs(off[i1])) if n not in (i0, i1))
        w = off[i0].copy()                                   # -k beta w_j of one row; its own entry from a second row
        w[i0] = off[i1, i0] * w[j] / off[i1, j]
        alpha = np.array([m[h, i, i] - (off[i, j] * w[i] / w[j] if i != j else off[i, i0] * w[i] / w[i0]) for i in range(D)])
        w /= np.linalg.norm(w / alpha)                       # w = a k, and k has length 1
        large = [r for r in range(0, D, 32) if abs(w[r]) > 1e-3]
        for col in range(D):
            r = large[col % len(large)]
            use = np.abs(w) > 2e-3
            use[r] = False
            a[h, r, col] = b[h, r, col] = np.float32(2.0 ** 8 * 1.02 / w[r])
            b[h, use, col] = (0.45 * 2.0 ** -15 / w[use]).astype(np.float32)
            grew[h, col] = (w * b[h, :, col]).sum() - w[r] * b[h, r, col]
            grew[h, col] /= w[r] * b[h, r, col]
        known.append((alpha, [i for i in np.argsort(-np.abs(off).max(axis=1)) if i not in large][:8]))
    sa, sb = step(a, b)
    return [np.median([((sb[h, i, col] - known[h][0][i] * b[h, i, col]) / sa[h, i, col] - 1.0) / grew[h, col] for col in range(D) for i in known[h][1]])
            for h in range(H)]


def test_sums_over_the_state_in_four_parts(gpu_lib):
    """An FP32 sum of all 32 rows of a thread keeps none of the 31 small ones, three quarters of a column's; four sums of eight rows lose
    seven, 0.94 of a column's are left. The threads' sums, the difference to v and the factor beta round by half a last place each, four
    where the small ones are 50 or more in all."""
    D, H = 128, 2
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.kda_head_dim, c.kda_heads, c.conv_k = 1, D, H, 4
    spec = synth.Spec(c, [0], [1], with_head=True)
    tensors = synth.make_model(spec, seed=17, recipe="spread")
    t = tensors["layers.0.self_attn.v_proj.weight"]
    tensors["layers.0.self_attn.v_proj.weight"] = (np.zeros_like(t[0]), t[1], t[2])
    eng, _ = common.build_models(spec, tensors, 32, oracle=False, options={"sequences": 2})

    def step(*states):
        eng.reset()
        for q, s in enumerate(states):
            eng.use_sequence(q)
            eng.state_write(0, 0, 0, s.astype(np.float32))
        eng.decode_batch(np.full(2, 5, np.int32))
        out = []
        for q in range(2):
            eng.use_sequence(q)
            out.append(eng.state_read(0, 0, 0, H * D * D).reshape(H, D, D).astype(np.float64))
        return out

    kept = _small_parts_kept(step, H, D)
    assert min(kept) > 0.94 - 4 / 50.0, kept
    eng.close()
