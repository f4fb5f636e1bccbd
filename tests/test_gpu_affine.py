"""The rotation kernel at the edges of its pieces of 32 pixels and bands of 16 rows, at rows off
a 16-byte boundary, at coordinates a hair below a whole number, and with windows and matrices that it
leaves to the pixel-by-pixel path.  Every byte against the oracle."""
import ctypes

import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


def _affine(oracle, img, m, th, tw):
    want = np.empty((th, tw, img.shape[2]), np.uint8)
    i64 = ctypes.c_int64
    oracle.lib().oracle_affine(oracle._p8(img), i64(img.shape[0]), i64(img.shape[1]), i64(img.shape[2]),
                               (ctypes.c_float * 6)(*m), i64(th), i64(tw), oracle._p8(want))
    return want


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (31, 16), (32, 17), (33, 15), (64, 4), (65, 33), (95, 18), (129, 5), (300, 40)])
def test_pieces(pkg, ctx, oracle, c, w, h):
    rng = np.random.default_rng(w * c)
    samples = [{"image": rng.integers(0, 256, (h + 9 + i, w + 11 + 2 * i, c), dtype=np.uint8)} for i in range(4)]
    for cast, gray in ((None, False), ((), False), (([0.4, 0.5, 0.6, 0.7][:c], [0.2, 0.3, 0.25, 0.5][:c]), False), ((), True)):
        if gray and c != 3:
            continue
        ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_rotate", dict(key="image", angle=float(13 + w), crop=True)),
               ("image_random_h_flip", dict(key="image", prob=0.5)), ("image_center_crop", dict(key="image", w=w, h=h))]
        if gray:
            ops.append(("image_channel_reduction", dict(key="image", preset="default")))
        arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
        oracle.set_state(c)
        want = oracle.run_chain(samples, ops, 4, {"image": 3.0}, arg)[0]["image"]
        oracle.set_state(c)
        got = chain.run_fused(pkg, ctx, samples, "image", ops, 4, cast, 3.0)[0]
        assert np.array_equal(got, want)


@pytest.mark.parametrize("cast", [None, ()])
def test_ragged_slots(pkg, ctx, oracle, cast):
    rng = np.random.default_rng(1)
    samples = [{"image": rng.integers(0, 256, (h, w, 3), dtype=np.uint8)} for h, w in ((70, 33), (5, 9), (31, 101), (64, 64))]
    ops = [("image_rotate", dict(key="image", angle=-27.0, crop=False))]
    want = oracle.run_chain(samples, ops, 4, {"image": 77.0}, None if cast is None else {"image": None})[0]["image"]
    assert np.array_equal(chain.run_fused(pkg, ctx, samples, "image", ops, 4, cast, 77.0)[0], want)


# a hair below a whole number the double sums of the definition round up to it; beside half ones they do not
@pytest.mark.parametrize("h,w,th,tw", [(9, 7, 8, 6), (9, 7, 9, 7), (8, 6, 8, 6), (33, 65, 40, 70)])
@pytest.mark.parametrize("hair", [-1e-20, -1e-9, -1.4e-8, -1.5e-8, -2.98e-8, -6e-8, 1e-20, -0.0])
def test_hairs(ctx, oracle, h, w, th, tw, hair):
    img = np.random.default_rng(3).integers(0, 256, (h, w, 3), dtype=np.uint8)
    for m in ((1, 0, hair, 0, 1, hair), (1, hair, -1, hair, 1, 2), (0, 1, hair, -1, 0, 0)):
        assert np.array_equal(ctx.image_affine(img, list(m), th, tw), _affine(oracle, img, m, th, tw))


@pytest.mark.parametrize("m", [(1, 0, 1e30, 0, 1, 0), (3e38, 3e38, -3e38, 1, 1, 0), (float("nan"), 0, 0, 0, 1, 0),
                               (1, 0, float("inf"), 0, 1, 0), (1e13, 0, 0, 0, 1, 0), (0, 0, 0, 0, 0, 0)])
def test_matrices_beyond(ctx, oracle, m):
    img = np.random.default_rng(4).integers(0, 256, (21, 40, 3), dtype=np.uint8)
    assert np.array_equal(ctx.image_affine(img, list(m), 30, 50), _affine(oracle, img, m, 30, 50))
