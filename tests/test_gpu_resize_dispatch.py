"""Which of the two resize kernels runs a batch: one of them all of it, but for batches
where the strong shrinks would flood the grid of the others, which take two launches.
Whichever it is, results are the oracle's."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


def _check(pkg, ctx, oracle, shapes, c, ops, seed, pad=5.0):
    rng = np.random.default_rng(seed)
    samples = [{"image": rng.integers(0, 256, (h, w, c), dtype=np.uint8)} for h, w in shapes]
    oracle.set_state(seed)
    want = [b["image"] for b in oracle.run_chain(samples, ops, len(samples), {"image": pad}, {"image": None})]
    oracle.set_state(seed)
    got = chain.run_fused(pkg, ctx, samples, "image", ops, len(samples), (), pad)
    assert len(want) == len(got) == 1 and np.array_equal(want[0], got[0])


# a wide and a tall shrink by 130 among many light ones: launches of their own
@pytest.mark.parametrize("c", [1, 3])
def test_two_launches(pkg, ctx, oracle, c):
    rng = np.random.default_rng(c)
    light = [(int(h), int(w)) for h, w in rng.integers(20, 61, (510, 2))]
    ops = [("image_resize", dict(key="image", w=64, h=64)), ("image_random_h_flip", dict(key="image", prob=0.5))]
    _check(pkg, ctx, oracle, light[:200] + [(64, 8320)] + light[200:300] + [(8320, 64)] + light[300:], c, ops, seed=c)


# the same with padding below the samples, which the first launch fills for both
def test_two_launches_of_ragged_slots(pkg, ctx, oracle):
    rng = np.random.default_rng(0)
    light = [(int(h), int(w)) for h, w in rng.integers(20, 61, (510, 2))]
    ops = [("image_resize_smallest_side", dict(key="image", size=40)), ("image_random_h_flip", dict(key="image", prob=0.5))]
    _check(pkg, ctx, oracle, light[:3] + [(4800, 4800)] + light[3:], 1, ops, seed=0)


# enough cells for the kernel of strong shrinks to be the faster one of two that can run them (two channels: the strips)
@pytest.mark.parametrize("c,side", [(1, 470), (2, 520), (3, 500), (4, 340)])
def test_large_batch_of_strong_shrinks(pkg, ctx, oracle, c, side):
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize", dict(key="image", w=100, h=98))]
    _check(pkg, ctx, oracle, [(side + i % 5, side - i % 7) for i in range(320)], c, ops, seed=c)


# either side of the lines (three to one, 13 / 3 down the rows, four channels), batches of a few images and of many
@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [2, 40])
def test_either_side_of_the_lines(pkg, ctx, oracle, c, n):
    for h, w in ((71, 209), (72, 210), (73, 211), (103, 200), (104, 200), (105, 200), (24 * 6, 70 * 4), (30, 90)):
        ops = [("image_resize", dict(key="image", w=70, h=24)), ("image_random_h_flip", dict(key="image", prob=0.5))]
        _check(pkg, ctx, oracle, [(h, w)] * n, c, ops, seed=c + n)
