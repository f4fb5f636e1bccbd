"""Resized batches cast by computed steps or, where those do not give the float32 chain of the
cast bit for bit, by the table: float batches against numpy's chain on the uint8 batch of the
same chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def four_channels(pkg):
    pkg.core.set_rgba_resize_independent(True)
    yield
    pkg.core.set_rgba_resize_independent(False)


CASTS = [dict(), dict(scale=1.0), dict(scale=3.7), dict(scale=-2.5e-39), dict(scale=1e38),
         dict(mean=[0.485, 0.456, 0.406, 0.5], std=[0.229, 0.224, 0.225, 0.25]),
         dict(scale=127.5, mean=[1.0, 0.0, -3.0, 7e7], std=[0.5, 3.0, 1e-30, 0.1]),
         dict(mean=[0.1, 0.2, 0.3, 0.4], std=[0.0, 1e38, 1e-45, 2.0])]   # infinities and NaN


@pytest.mark.parametrize("cast", range(len(CASTS)))
@pytest.mark.parametrize("c,size", [(1, 37), (2, 48), (3, 64), (4, 33), (3, 300), (1, 300), ("gray", 50)])
def test_float_batch_is_the_cast_of_the_byte_batch(pkg, c, size, cast):
    rng = np.random.default_rng(5)
    gray, ch = c == "gray", 3 if c == "gray" else c
    shapes = [(100, 90), (70, 210), (150, 64)]
    samples = [{"image": rng.integers(0, 256, (h, w, ch), dtype=np.uint8)} for h, w in shapes]
    kw = dict(CASTS[cast])
    co = 1 if gray else ch
    for k in ("mean", "std"):
        if k in kw:
            kw[k] = kw[k][:co]
    ds = pkg.buffer_from_vector(samples).image_resize("image", size, size - 5)
    if gray:
        ds = ds.image_channel_reduction("image", "default")
    ds = ds.batch(len(samples))
    raw = ds[0]["image"]
    with np.errstate(all="ignore"):
        want = raw.astype(np.float32) / np.float32(kw.get("scale", 255))
        if "mean" in kw:
            want = (want - np.float32(kw["mean"])) / np.float32(kw["std"])
    got = ds.key_cast("image", **kw)[0]["image"]
    assert got.dtype == np.float32 and np.array_equal(got.view(np.uint32), want.view(np.uint32)) or \
        np.array_equal(got, want, equal_nan=True)
