"""Float batches bit for bit: every value that is not NaN has the bits of numpy's float32 chain on
the byte batch (a zero's sign among them), NaN stand where numpy has them, and those that a NaN in the
cast gives are that NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAN = float("nan")
CASTS = [dict(), dict(scale=3.7), dict(scale=1e38), dict(mean=[0.485, 0.456, 0.406, 0.5], std=[0.229, 0.224, 0.225, 0.25]),
         dict(mean=[0.0, -0.0, 0.5, 1.0], std=[-0.25, -3.0, -1e30, 1e38]), dict(mean=[0.1, 0.2, 0.3, 0.4], std=[0.0, 1e38, 1e-45, 2.0]),
         dict(mean=[0.1, 0.2, 0.3, 0.4], std=[0.5, NAN, 0.25, 0.5])]


@pytest.mark.parametrize("cast", range(len(CASTS)))
@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("chain", ["shrink", "enlarge", "copy", "rotate"])
def test_bits(pkg, chain, c, cast):
    rng = np.random.default_rng(c)
    samples = [{"image": rng.integers(0, 256, (h, w, c), dtype=np.uint8)} for h, w in ((100, 90), (70, 210), (150, 64))]
    samples[0]["image"][:40] = 0
    kw = {k: v if k == "scale" else v[:c] for k, v in CASTS[cast].items()}
    pkg.core.set_rgba_resize_independent(True)
    try:
        ds = pkg.buffer_from_vector(samples)
        if chain == "rotate":
            ds = ds.image_rotate("image", angle=33.0, crop=False)
        elif chain != "copy":
            ds = ds.image_resize("image", *((37, 31) if chain == "shrink" else (300, 290)))
        ds = ds.batch(len(samples))
        raw = ds[0]["image"]
        got = ds.key_cast("image", **kw)[0]["image"]
    finally:
        pkg.core.set_rgba_resize_independent(False)
    with np.errstate(all="ignore"):
        want = raw.astype(np.float32) / np.float32(kw.get("scale", 255))
        if "mean" in kw:
            want = (want - np.float32(kw["mean"])) / np.float32(kw["std"])
    assert got.dtype == np.float32 and got.shape == want.shape
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    bits, expected = got.view(np.uint32), want.view(np.uint32)
    assert np.array_equal(bits[~nan], expected[~nan])
    for ch in range(c):
        if "std" in kw and np.isnan(kw["std"][ch]):
            assert (bits[..., ch] == np.float32(kw["std"][ch]).view(np.uint32)).all()
