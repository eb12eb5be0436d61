"""The indexer's pool scores (csrc/mla.cu): the tiled kernel has the same bits as the one that takes any shape, whose sums are the
reference's, heads and dimensions ascending (src/core/glm53f_dsa.c:141-157)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim", [(8, 16), (8, 48), (16, 112), (24, 128), (32, 128), (32, 256), (24, 208)])
def test_both_kernels_give_the_same_bits(gpu_lib, heads, dim):
    """Part of a tile of 64 pools, whole ones and one more; a warp's 16 pools; several queries; scores spread over many binades."""
    rng = np.random.default_rng(heads * dim)
    for pools, T in ((1, 1), (15, 1), (16, 2), (63, 3), (64, 1), (65, 1), (200, 17), (1000, 3)):
        keys = (rng.standard_normal((pools + T - 1, dim)) * np.exp2(rng.integers(-12, 13, (pools + T - 1, 1)))).astype(np.float32)
        q, w = rng.standard_normal((T, heads, dim)).astype(np.float32), rng.standard_normal((T, heads)).astype(np.float32)
        got = [np.empty((T, pools + T + 1), np.float32) for _ in range(2)]
        for tiled in (0, 1):
            assert gpu_lib.g5b_debug_dsa_scores(keys.ctypes.data, pools, q.ctypes.data, w.ctypes.data, T, heads, dim, tiled, got[tiled].ctypes.data, 0) == 0
        assert np.array_equal(got[0], got[1]), (pools, T)
        dots = np.einsum("thd,pd->thp", q.astype(np.float64), keys.astype(np.float64)) / np.sqrt(dim)
        want = np.einsum("th,thp->tp", w.astype(np.float64), np.maximum(dots, 0.0)) / np.sqrt(heads)
        size = np.einsum("th,thp->tp", np.abs(w).astype(np.float64), np.maximum(dots, 0.0)) / np.sqrt(heads)
        seen = np.arange(pools + T - 1)[None] < pools + np.arange(T)[:, None]
        # five roundings to floats, half a place each: the square root and the quotient of either scale factor, the sum
        assert (np.abs(got[1][:, :pools + T - 1] - want)[seen] <= 5 * 2.0 ** -24 * size[seen] + 1e-30).all()
        assert np.abs(got[1][:, :pools + T - 1][~seen]).max(initial=0.0) == 0.0
