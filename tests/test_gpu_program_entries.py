"""Keys of a sample while its ops are recorded as programs: an op into another key leaves its
input as it was, one in place replaces it, a program that is full is computed and a new one
begun, and what an op reads from another key is that key's array."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _samples(n=5):
    rng = np.random.default_rng(8)
    return [{"image": rng.integers(0, 256, (40 + i, 50 - i, 3), dtype=np.uint8), "angle": np.float64(90.0 * (i % 4))}
            for i in range(n)]


def _crop(a, w, h):
    y, x = (a.shape[0] - h) // 2, (a.shape[1] - w) // 2
    return a[y:y + h, x:x + w]


@pytest.mark.parametrize("kind", ["buffer", "stream"])
def test_output_keys(pkg, kind):
    samples = _samples()
    ds = pkg.buffer_from_vector(samples)
    ds = ds if kind == "buffer" else ds.to_stream()
    ds = ds.image_center_crop("image", 20, 16, output_key="b").image_random_h_flip("image", 1.0)
    ds = ds.image_random_h_flip("b", 1.0, output_key="c").image_center_crop("b", 10, 8)
    ds = ds.image_center_crop("image", 24, 20).image_center_crop("c", 12, 6, output_key="image2")
    got = next(iter(ds.batch(5)))
    for i, s in enumerate(samples):
        b = _crop(s["image"], 20, 16)
        assert np.array_equal(got["image"][i], _crop(s["image"][:, ::-1], 24, 20))
        assert np.array_equal(got["b"][i], _crop(b, 10, 8))
        assert np.array_equal(got["c"][i], b[:, ::-1])
        assert np.array_equal(got["image2"][i], _crop(b[:, ::-1], 12, 6))


def test_full_programs(pkg):
    samples = _samples()
    ds = pkg.buffer_from_vector(samples)
    # padding takes no crop: computed, then a new program, in the same key and in another
    ds = ds.pad("image", 1, 0, 6, 7.0).image_center_crop("image", 30, 30, output_key="b")
    ds = ds.image_center_crop("image", 28, 26).pad("b", 0, 2, 0, 3.0)
    got = ds.batch(5)[0]
    for i, s in enumerate(samples):
        p = np.pad(s["image"], ((0, 0), (0, 6), (0, 0)), constant_values=7)
        assert np.array_equal(got["image"][i], _crop(p, 28, 26))
        assert np.array_equal(got["b"][i], np.pad(_crop(p, 30, 30), ((2, 0), (0, 0), (0, 0)), constant_values=3))


def test_read_keys(pkg, oracle):
    samples = _samples(4)
    want = [oracle.rotate(s["image"], float(s["angle"]), True) for s in samples]
    ds = pkg.buffer_from_vector(samples).image_rotate("image", 0.0, crop=True, angle_key="angle", output_key="angle")
    ds = ds.image_center_crop("image", 30, 30)
    got = ds.batch(4)[0]
    for i, s in enumerate(samples):
        h, w = want[i].shape[:2]
        assert np.array_equal(got["angle"][i][:h, :w], want[i])
        assert np.array_equal(got["image"][i], _crop(s["image"], 30, 30))
    with pytest.raises(RuntimeError):
        pkg.buffer_from_vector(samples).image_rotate("image", 0.0, crop=True, angle_key="none").batch(4)[0]
