"""Sources in ordinary host memory, packed by the calling threads and copied while others are
still being packed: rows shorter and longer than what leaves at a time, whole images and
windows of them, batches below and above the size that is sent in parts, and such sources beside
page-locked ones.  Every byte against the oracle; the lane's block is used again at once."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,crop", [((3, 1, 1), (1, 2)), ((40, 21, 1), (21, 40)), ((33, 64, 1), (64, 33)), ((50, 85, 3), (61, 44)),
                                        ((70, 64, 4), (63, 70)), ((90, 300, 3), (256, 80)), ((1100, 700, 3), (600, 900)),
                                        ((1300, 1900, 3), (1900, 1300))])
@pytest.mark.parametrize("n", [1, 3, 9])
def test_packed_sources(pkg, ctx, oracle, shape, crop, n):
    rng = np.random.default_rng(n)
    ops = [("image_random_crop", dict(key="image", w=crop[0], h=crop[1])), ("image_random_h_flip", dict(key="image", prob=0.5))]
    for seed in range(3):
        samples = [{"image": rng.integers(0, 256, shape, dtype=np.uint8)} for _ in range(n)]
        oracle.set_state(seed)
        want = oracle.run_chain(samples, ops, n, {"image": 0.0}, None)[0]["image"]
        oracle.set_state(seed)
        assert np.array_equal(chain.run_fused(pkg, ctx, samples, "image", ops, n)[0], want)


def test_beside_page_locked_sources(pkg, oracle):
    rng = np.random.default_rng(2)
    samples = []
    for i in range(8):
        a = rng.integers(0, 256, (800 + 7 * i, 900 - 11 * i, 3), dtype=np.uint8)
        if i % 3 == 1:
            held = pkg.core.pinned_empty(list(a.shape), "uint8")
            held[...] = a
            a = held
        samples.append({"image": a})
    ops = [("image_resize_smallest_side", dict(key="image", size=300)), ("image_center_crop", dict(key="image", w=299, h=300))]
    ds = pkg.buffer_from_vector(samples)
    for op, kw in ops:
        ds = getattr(ds, op)(**kw)
    want = oracle.run_chain([{"image": np.array(s["image"])} for s in samples], ops, 8, {"image": 0.0}, None)[0]["image"]
    for _ in range(3):
        assert np.array_equal(ds.batch(8)[0]["image"], want)
