"""Mirrored crops whose width is no multiple of four: the last group of four
pixels of a row is partly empty, and its empty places index nothing."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 2, 3, 5, 29, 30, 31, 33, 65])
@pytest.mark.parametrize("c", [1, 3, 4])
def test_mirrored_crop_of_any_width(pkg, ctx, oracle, width, c):
    rng = np.random.default_rng(7 * width + c)
    samples = [{"image": rng.integers(0, 256, (40, 80 + i, c), dtype=np.uint8)} for i in range(3)]
    ops = [("image_random_h_flip", dict(key="image", prob=1.0)), ("image_center_crop", dict(key="image", w=width, h=21))]
    for cast in (None, (), ([0.4] * c, [0.2] * c)):
        arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
        oracle.set_state(3)
        want = [b["image"] for b in oracle.run_chain(samples, ops, 3, {"image": 9.0}, arg)]
        oracle.set_state(3)
        got = chain.run_fused(pkg, ctx, samples, "image", ops, 3, cast, 9.0)
        assert len(want) == len(got) and all(np.array_equal(w, g) for w, g in zip(want, got))
