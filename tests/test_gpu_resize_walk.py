"""The resize kernel where its split can go wrong: chunk and stage borders, row
pitches of every residue mod 4, windows that start at any byte, enlargements,
ratios whose taps meet in one source row, shrinks up to and beyond one chunk,
mirrors on either side.  The oracle performs the same float32 operations in the
same order, so results are equal."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


def _check(pkg, ctx, oracle, shapes, c, ops, cast=(), seed=0):
    rng = np.random.default_rng(seed)
    samples = [{"image": rng.integers(0, 256, (h, w, c), dtype=np.uint8)} for h, w in shapes]
    arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
    oracle.set_state(seed)
    want = [b["image"] for b in oracle.run_chain(samples, ops, len(samples), {"image": 7.0}, arg)]
    oracle.set_state(seed)
    got = chain.run_fused(pkg, ctx, samples, "image", ops, len(samples), cast, 7.0)
    assert len(want) == len(got) == 1 and np.array_equal(want[0], got[0])


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("out", [(1, 1), (3, 127), (4, 128), (5, 129), (31, 64), (32, 300), (33, 257), (70, 2)])
def test_output_sizes(pkg, ctx, oracle, c, out):
    shapes = [(97, 200), (64, 201), (33, 202), (150, 203), (300, 77), (out[0], 90), (80, out[1] + 1), (1, 1), (2, 3)]
    ops = [("image_resize", dict(key="image", w=out[1], h=out[0]))]
    _check(pkg, ctx, oracle, shapes, c, ops, cast=None if out[1] % 2 else ())


@pytest.mark.parametrize("ratio", [1.0 / 7, 0.5, 1.01, 2.0, 3.0, 5.0, 8.0 / 3, 24.0, 90.0, 150.0])
@pytest.mark.parametrize("flip", ["none", "before", "after"])
def test_ratios(pkg, ctx, oracle, ratio, flip):
    h, w = 37, 41
    shapes = [(max(1, round(h * ratio)), max(1, round(w * ratio) + k)) for k in range(2 if ratio > 20 else 4)]
    mirror = [("image_random_h_flip", dict(key="image", prob=1.0))]
    ops = [("image_resize", dict(key="image", w=w, h=h))]
    ops = mirror + ops if flip == "before" else ops + mirror if flip == "after" else ops
    _check(pkg, ctx, oracle, shapes, 3, ops, cast=([0.4, 0.5, 0.6], [0.2, 0.3, 0.25]))


@pytest.mark.parametrize("cut", range(4))
@pytest.mark.parametrize("c", [1, 3, 4])
def test_windows_at_any_byte(pkg, ctx, oracle, cut, c):
    ops = [("image_center_crop", dict(key="image", w=160 + cut, h=90)), ("image_resize", dict(key="image", w=140, h=50)),
           ("image_center_crop", dict(key="image", w=133 - cut, h=35 + cut))]
    if c == 3:
        ops.append(("image_channel_reduction", dict(key="image", preset="rec709")))
    _check(pkg, ctx, oracle, [(120, 190), (120, 191), (121, 192), (90, 193)], c, ops, seed=cut)
