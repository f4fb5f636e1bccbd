"""key_cast after batch into a key that the samples have already: the cast comes
later in the chain, so its output is what the key holds, whatever the keys are
called."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ["image", "label", "a", "b"]


def _samples(names):
    rng = np.random.default_rng(4)
    return [{k: rng.integers(0, 256, (9, 11, 3), dtype=np.uint8) for k in names} for _ in range(5)]


@pytest.mark.parametrize("source,target", list(itertools.permutations(KEYS, 2)))
@pytest.mark.parametrize("kind", ["buffer", "stream"])
def test_cast_replaces_the_key_it_names(pkg, source, target, kind):
    samples = _samples((source, target))
    ds = pkg.buffer_from_vector(samples)
    ds = ds if kind == "buffer" else ds.to_stream()
    batches = [b for b in ds.batch(5).key_cast(source, output_key=target)]
    raw = np.stack([s[source] for s in samples])
    assert len(batches) == 1 and set(batches[0]) == {source, target}
    assert np.array_equal(batches[0][source], raw)
    assert np.array_equal(batches[0][target], raw.astype(np.float32) / np.float32(255))


def test_casts_apply_in_the_order_they_were_written(pkg):
    samples = _samples(KEYS)
    x = {k: np.stack([s[k] for s in samples]) for k in KEYS}
    ds = pkg.buffer_from_vector(samples).batch(5)
    for k in ("b", "image", "a"):
        ds = ds.key_cast(k, output_key="label")
    got = ds.key_cast("b", scale=51.0)[0]
    assert np.array_equal(got["label"], x["a"].astype(np.float32) / np.float32(255))
    assert np.array_equal(got["b"], x["b"].astype(np.float32) / np.float32(51))
    assert np.array_equal(got["a"], x["a"]) and np.array_equal(got["image"], x["image"])


def test_cast_of_arrays_that_are_no_images(pkg):
    rng = np.random.default_rng(4)
    samples = [{k: rng.integers(0, 256, (7, 3), dtype=np.uint8) for k in KEYS} for _ in range(3)]
    for source, target in itertools.permutations(KEYS, 2):
        got = pkg.buffer_from_vector(samples).batch(3).key_cast(source, output_key=target)[0]
        want = np.stack([s[source] for s in samples])
        assert np.array_equal(got[source], want)
        assert np.array_equal(got[target], want.astype(np.float32) / np.float32(255))
