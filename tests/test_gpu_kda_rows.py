"""Several positions of one sequence (csrc/kda.cu): the preparation's tiles of 16 positions and the scan's groups of 8, both head
sizes, convolutions of the known and of another width; and the sigmoid by pairs that the preparation takes."""
import numpy as np
import pytest

import common
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim,heads,conv", [(128, 3, 4), (64, 5, 4), (128, 2, 3), (64, 2, 1)])
def test_prompts_around_the_tiles(gpu_lib, binding, head_dim, heads, conv):
    """Calls that end at, before and behind a tile, each with the history that the one before it left (1e-5: 35 positions whose sums of
    128 products are taken in another order, 2^-24 * sqrt(128) each, and a norm over them)."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.kda_head_dim, c.kda_heads, c.conv_k = 2, head_dim, heads, conv
    spec = synth.Spec(c, [0, 0], [1, 1], with_head=True)
    tensors = synth.make_model(spec, seed=12, recipe="spread")
    eng, orc = common.build_models(spec, tensors, 128, binding)
    rng = np.random.default_rng(3)
    for T in (2, 15, 16, 17, 35, 3):
        x = rng.standard_normal((T, c.hidden)).astype(np.float32)
        assert common.rel_err(eng.op_kda(0, x), orc.op_kda(0, x)) < 1e-5, T
    n = heads * head_dim ** 2 + 3 * heads * head_dim * (conv - 1)
    assert common.rel_err(eng.state_read(0, 0, 0, n), orc.state_read(0, 0, 0, n)) < 1e-5
    eng.close()
    orc.close()


def test_sigmoid_by_pairs_is_the_rounded_quotient(gpu_lib):
    """Bit for bit 1 / (1 + e) of the single exponential e, as long as the quotient is a normal number; 1, 0 and NaN at the ends."""
    rng = np.random.default_rng(4)
    x = np.concatenate([np.linspace(-87, 104, 1 << 20), rng.standard_normal(1 << 20) * 4, [np.inf, -np.inf, np.nan, 200.0, -200.0]]).astype(np.float32)
    e, s, minus = np.empty_like(x), np.empty_like(x), np.ascontiguousarray(-x)
    assert gpu_lib.g5b_debug_exp(minus.ctypes.data, x.size, e.ctypes.data, s.ctypes.data, 0) == 0        # e = exp(-x)
    unused = np.empty_like(x)
    assert gpu_lib.g5b_debug_exp(x.ctypes.data, x.size, unused.ctypes.data, s.ctypes.data, 0) == 0
    assert np.array_equal(s, (np.float32(1) / (np.float32(1) + e)).astype(np.float32), equal_nan=True)


def test_reciprocal_of_every_mantissa(gpu_lib):
    """Arguments whose 1 + exp(-x) runs through all 2^23 floats from 1 to 2: x is off by half of its last place and the exponential by
    0.53 of its own, together less than half the distance of two of these sums. Bit for bit the divided ones."""
    n = 1 << 23
    x = np.full(n, 200.0, np.float32)
    x[1:] = -np.log(np.arange(1, n) / n)
    minus, e, s, unused = -x, np.empty_like(x), np.empty_like(x), np.empty_like(x)
    assert gpu_lib.g5b_debug_exp(minus.ctypes.data, n, e.ctypes.data, unused.ctypes.data, 0) == 0
    assert gpu_lib.g5b_debug_exp(x.ctypes.data, n, unused.ctypes.data, s.ctypes.data, 0) == 0
    d = np.float32(1) + e
    assert np.array_equal(d.view(np.uint32), np.arange(n, dtype=np.uint32) + np.float32(1).view(np.uint32))
    assert np.array_equal(s, np.float32(1) / d)
