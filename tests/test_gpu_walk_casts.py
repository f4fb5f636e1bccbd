"""Shrinks that resize_walk.cu runs, in every way that it stores: bytes, floats cast by either kind of
steps, through the table (a cast with infinities, one with a NaN) and behind the channel reduction.
Rows of whole words and others in one batch, like and unlike samples, padded and full slots.  Bytes against
the oracle, floats bit for bit against numpy's chain on them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASTS = [dict(), dict(scale=1e-40), dict(mean=[0.485, 0.456, 0.406, 0.5], std=[0.229, 0.224, 0.225, 0.25]),
         dict(mean=[0.1, 0.2, 0.3, 0.4], std=[0.5, float("nan"), 0.25, 0.5])]
SHAPES = {"like": [(301, 420)] * 5, "odd": [(300, 333)] * 3, "unlike": [(301, 420), (640, 201), (96, 800), (333, 257), (700, 340), (64, 64)],
          "own": [(2400, 60), (60, 2400), (61, 90), (120, 64)]}


@pytest.fixture(autouse=True)
def four_channels(pkg):
    pkg.core.set_rgba_resize_independent(True)
    yield
    pkg.core.set_rgba_resize_independent(False)


@pytest.mark.parametrize("shapes", sorted(SHAPES))
@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("c", [1, 2, 3, 4, "gray"])
def test_ways_of_storing(pkg, oracle, c, padded, shapes):
    rng = np.random.default_rng(11)
    ch, co = (3, 1) if c == "gray" else (c, c)
    samples = [{"image": rng.integers(0, 256, (h, w, ch), dtype=np.uint8)} for h, w in SHAPES[shapes]]
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)),
           ("image_resize_smallest_side", dict(key="image", size=9)) if padded else ("image_resize", dict(key="image", w=13, h=11)),
           ("image_random_h_flip", dict(key="image", prob=0.5))]
    if c == "gray":
        ops.append(("image_channel_reduction", dict(key="image", preset="default")))
    n = len(samples)
    oracle.set_state(7)
    want = oracle.run_chain(samples, ops, n, {"image": 5.0})[0]["image"]
    ds = pkg.buffer_from_vector(samples)
    for op, kw in ops:
        ds = getattr(ds, op)(**kw)
    ds = ds.batch(n, pad={"image": 5.0})
    pkg.core.set_state(7)
    assert np.array_equal(ds[0]["image"], want)
    for cast in CASTS:
        kw = {k: v if k == "scale" else v[:co] for k, v in cast.items()}
        pkg.core.set_state(7)
        got = ds.key_cast("image", **kw)[0]["image"]
        with np.errstate(all="ignore"):
            floats = want.astype(np.float32) / np.float32(kw.get("scale", 255))
            if "mean" in kw:
                floats = (floats - np.float32(kw["mean"])) / np.float32(kw["std"])
        nan = np.isnan(floats)
        assert got.dtype == np.float32 and np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint32)[~nan], floats.view(np.uint32)[~nan])
