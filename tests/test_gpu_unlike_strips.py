"""Batches whose samples have their largest needs of shared memory in different places - wide
strips of enlargements, rows in flight and steps of strong shrinks, many taps - each strip laid out
for its own.  Every byte against the oracle."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("n,size", [(5, 40), (5, 257), (70, 96), (70, 224)])
@pytest.mark.parametrize("cast", [None, ()])
def test_unlike_samples(pkg, ctx, oracle, c, n, size, cast):
    rng = np.random.default_rng(n + c)
    shapes = [(int(size * rng.uniform(0.1, 6.3)), int(size * rng.choice([0.2, 1.0, 2.0, 3.9]))) for _ in range(n)]
    shapes[0], shapes[1], shapes[2] = (size * 6, size), (size, size * 4), (max(2, size // 8), max(2, size // 8))
    samples = [{"image": rng.integers(0, 256, (max(1, h), max(1, w), c), dtype=np.uint8)} for h, w in shapes]
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize", dict(key="image", w=size, h=size + 3))]
    oracle.set_state(1)
    want = oracle.run_chain(samples, ops, n, {"image": 0.0}, None if cast is None else {"image": None})[0]["image"]
    oracle.set_state(1)
    assert np.array_equal(chain.run_fused(pkg, ctx, samples, "image", ops, n, cast)[0], want)
