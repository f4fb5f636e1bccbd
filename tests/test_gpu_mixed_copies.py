"""Batches in which some images have the size of the resize already: a few become resizes by
1 beside the others, more keep a launch of their own (launch_plan.cu: join_copies).  Every
byte against the oracle."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("copies,others,side", [(1, 5, 61), (3, 3, 256), (1, 1, 700), (40, 3, 300)])
@pytest.mark.parametrize("cast", [None, (), "flip"])
def test_copies_among_resizes(pkg, ctx, oracle, c, copies, others, side, cast):
    rng = np.random.default_rng(copies * 10 + c)
    shapes = [(side, side + int(rng.integers(0, 30))) for _ in range(copies)]
    shapes += [(int(rng.integers(side // 2, 3 * side)), int(rng.integers(side // 2, 3 * side))) for _ in range(others)]
    rng.shuffle(shapes)
    samples = [{"image": rng.integers(0, 256, (h, w, c), dtype=np.uint8)} for h, w in shapes]
    ops = [("image_resize_smallest_side", dict(key="image", size=side)),
           ("image_center_crop", dict(key="image", w=side - 7, h=side - 4))]
    if cast == "flip":
        ops = [("image_random_h_flip", dict(key="image", prob=0.5))] + ops + [("image_random_h_flip", dict(key="image", prob=0.5))]
        cast = None
    arg = None if cast is None else {"image": None}
    oracle.set_state(3)
    want = [b["image"] for b in oracle.run_chain(samples, ops, len(samples), {"image": 9.0}, arg)]
    oracle.set_state(3)
    got = chain.run_fused(pkg, ctx, samples, "image", ops, len(samples), cast=cast, pad=9.0)
    assert len(want) == len(got) == 1 and np.array_equal(want[0], got[0])
