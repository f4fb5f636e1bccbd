"""The line between the resize kernel and the one that filters pixel by pixel: a
column whose taps and words take more than 832 source bytes, or a row of more
than 1024 steps, is the latter's.  Both do the oracle's float32 operations in its
order, so results are equal on either side of the line; a plan that put a sample
into the resize kernel beyond its room would be refused by the kernel's check."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu

# the strongest shrink along a row, in source columns to three, whose 2r + 2 columns fit 826 bytes
LAST_WIDTH = {1: 1236, 2: 616, 3: 409, 4: 306}
# and down the rows: 2r + 11 steps within 1024
LAST_HEIGHT = 1519


def _check(pkg, ctx, oracle, shapes, c, ops, seed):
    rng = np.random.default_rng(seed)
    samples = [{"image": rng.integers(0, 256, (h, w, c), dtype=np.uint8)} for h, w in shapes]
    gray = any(name == "image_channel_reduction" for name, _ in ops)
    co = 1 if gray else c
    for cast in (None, (), ([0.4] * co, [0.2] * co)):
        arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
        oracle.set_state(seed)
        want = [b["image"] for b in oracle.run_chain(samples, ops, len(samples), {"image": 9.0}, arg)]
        oracle.set_state(seed)
        got = chain.run_fused(pkg, ctx, samples, "image", ops, len(samples), cast, 9.0)
        assert len(want) == len(got) == 1 and np.array_equal(want[0], got[0])


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("beyond", [0, 1, 2])
def test_limit_along_a_row(pkg, ctx, oracle, c, beyond):
    w = LAST_WIDTH[c] + beyond
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize", dict(key="image", w=3, h=9))]
    _check(pkg, ctx, oracle, [(14, w), (9, w + 1), (5, w), (12, 40), (9, 3)], c, ops, seed=c + beyond)


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("beyond", [0, 1, 2])
def test_limit_down_the_rows(pkg, ctx, oracle, c, beyond):
    h = LAST_HEIGHT + beyond
    ops = [("image_resize", dict(key="image", w=10, h=3)), ("image_random_h_flip", dict(key="image", prob=0.5))]
    _check(pkg, ctx, oracle, [(h, 14), (h + 1, 10), (h, 7), (40, 12), (3, 10)], c, ops, seed=c + beyond)


@pytest.mark.parametrize("beyond", [0, 1])
@pytest.mark.parametrize("axis", ["x", "y"])
def test_limits_with_the_channel_reduction(pkg, ctx, oracle, beyond, axis):
    w, h, shape = (3, 9, (14, LAST_WIDTH[3] + beyond)) if axis == "x" else (10, 3, (LAST_HEIGHT + beyond, 14))
    ops = [("image_resize", dict(key="image", w=w, h=h)), ("image_channel_reduction", dict(key="image", preset="rec601"))]
    _check(pkg, ctx, oracle, [shape, (20, 30)], 3, ops, seed=beyond)


@pytest.mark.parametrize("c", [1, 2, 3, 4])
def test_far_beyond_both_in_ragged_slots(pkg, ctx, oracle, c):
    """Windows, mirrors, padding beside and below; samples of both kernels and of the copy in one batch."""
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize_smallest_side", dict(key="image", size=3)),
           ("image_random_h_flip", dict(key="image", prob=0.5))]
    _check(pkg, ctx, oracle, [(1700, 1700), (1700, 2300), (5, 3), (40, 70), (3, 8), (1530, 1280)], c, ops, seed=c)


# (along which axis, source and result, channels): the planner's bounds have to hold float32 positions that
# are a sample or two off at this distance from the image's edge
@pytest.mark.parametrize("axis,n,m,c", [("y", 9716434, 8426337, 1), ("y", 9489329, 6289399, 1), ("y", 8597653, 3954443, 1),
                                        ("x", 8865487, 9554784, 3), ("x", 9446063, 2688457, 3)])
def test_sides_beyond_the_integers_of_float32(pkg, oracle, axis, n, m, c):
    img = np.random.default_rng(n).integers(0, 256, (n, 2, c) if axis == "y" else (2, n, c), dtype=np.uint8)
    w, h = (2, m) if axis == "y" else (m, 2)
    own = pkg.Context(device=0, n_lanes=1)
    try:
        got = own.image_resize(img, w, h)
    finally:
        own.close()
    assert np.array_equal(got, oracle.resize(img, w, h))
