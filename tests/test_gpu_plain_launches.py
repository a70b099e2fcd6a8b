"""Only decoding steps chain their kernels: in a pass with a prompt every kernel up to the gather of the wanted rows is launched plainly, also
those over a few of its rows (the single tokens beside the prompt)."""
import numpy as np
import pytest

from test_gpu_flash import LATENT
from test_gpu_mixed_attention import config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,singles", [(config(128, 16, 50.0), 10), (LATENT, 3)])
def test_dependent_launches_of_each_kind_of_pass(model, singles):
    from kapel_b200 import kernels as K
    from kapel_b200.engine import Engine

    rng = np.random.default_rng(4)
    eng = Engine.random(model, seed=1, dtype="bfloat16", max_tokens=singles * 64 + 512, max_sequences=singles + 1, graphs=False)
    draw = lambda n: rng.integers(0, 90, n).tolist()
    ones = lambda: [(f"s{i}", draw(1), [0]) for i in range(singles)]

    norm, at_tail = eng.model.final_norm.forward, []
    eng.model.final_norm.forward = lambda x: at_tail.append(K.dependent_launch_count()) or norm(x)

    def chained(entries):
        before = K.dependent_launch_count()
        eng.step(entries)
        return at_tail[-1] - before

    assert chained([(f"s{i}", draw(30), [29]) for i in range(singles)]) == 0
    assert chained(ones() + [("p", draw(100), [99])]) == 0
    assert (chained(ones()) > 0) == K.PDL
    assert chained([("p", draw(70), [3, 69])]) == 0
    eng.check()


@pytest.mark.parametrize("model,singles", [(config(128, 16, 50.0), 10), (LATENT, 3)])
def test_mixed_passes_with_poisoned_buffers(model, singles):
    """Every buffer of a pass cut in two is one that the poisoning mode fills: the logits are the same with it, bit for bit."""
    from kapel_b200 import kernels as K
    from kapel_b200.engine import Engine

    eng = Engine.random(model, seed=1, dtype="bfloat16", max_tokens=2 * singles * 64 + 1024, max_sequences=2 * (singles + 1), graphs=False)
    made, kept, got = [], K._fresh, []
    for turn in "ab":
        rng = np.random.default_rng(4)
        draw = lambda n: rng.integers(0, 90, n).tolist()
        eng.step([(f"{turn}{i}", draw(30), []) for i in range(singles)])
        K.set_poison(turn == "b")
        K._fresh = lambda shape, *rest: made.append(tuple(shape)) or kept(shape, *rest)
        try:
            got.append(eng.step([(f"{turn}{i}", draw(1), [0]) for i in range(singles)] + [(turn, draw(100), [5, 99])]).cpu())
        finally:
            K.set_poison(False)
            K._fresh = kept
    assert np.isfinite(got[0].numpy()).all() and (got[0] == got[1]).all()
    # the whole pass's attention output, which its two halves write: beside the queries in two layers, alone in one; both turns
    whole, times = ((singles + 100, 32, 128), 8) if model is not LATENT else ((singles + 100, 3 * 128), 2)
    assert made.count(whole) == times
