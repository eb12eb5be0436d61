"""The arg-max of a row of logits (csrc/elementwise.cu): parts of one element, of a few, of several rounds of eight; equal logits."""
import numpy as np
import pytest

import common
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [40, 64, 1000, 131200])
def test_first_of_the_largest_logits(gpu_lib, vocab):
    """Every second row of the head repeats the one before it, so that each logit is there twice: the lower index wins. A call that wants no
    arg-max leaves the next one's right."""
    c = synth.tiny_spec().cfg.copy()
    c.n_layers, c.vocab = 1, vocab
    spec = synth.Spec(c, [0], [1], with_head=True)
    tensors = synth.make_model(spec, seed=41, recipe="spread")
    head = tensors["lm_head.weight"][0]
    head[1::2] = head[0::2]
    eng, _ = common.build_models(spec, tensors, 32, oracle=False)
    for ids in ([1, 5, 3], [7], [2]):
        logits, am = eng.forward(np.array(ids, np.int32), want_logits=True, want_argmax=len(ids) != 1 or ids[0] == 2)
        if am is not None:
            assert am[-1] == int(np.argmax(logits)) and am[-1] % 2 == 0
    first = int(np.argmax(logits))
    assert len(eng.decode_greedy(first, 3)) == 3
    eng.close()
