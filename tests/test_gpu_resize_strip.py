"""The lines between the resize kernels: a strip of 241 source bytes holds too few
columns of a strong shrink along a row, 14 source rows do not hold one output row of a
strong shrink down the rows (or four, or two of them, which then come in parts).  Both
kernels do the oracle's float32 operations in its order, so results are equal on either
side; rows of every pitch and first byte, mirrors, ragged slots, kernels mixed in a batch."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


def _check(pkg, ctx, oracle, shapes, c, ops, seed, casts=(None, ())):
    rng = np.random.default_rng(seed)
    samples = [{"image": rng.integers(0, 256, (h, w, c), dtype=np.uint8)} for h, w in shapes]
    for cast in casts:
        arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
        oracle.set_state(seed)
        want = [b["image"] for b in oracle.run_chain(samples, ops, len(samples), {"image": 5.0}, arg)]
        oracle.set_state(seed)
        got = chain.run_fused(pkg, ctx, samples, "image", ops, len(samples), cast, 5.0)
        assert len(want) == len(got) == 1 and np.array_equal(want[0], got[0])


# down the rows: 5r, 3r and 2r + 2 source rows against 14, at 20 output rows
@pytest.mark.parametrize("h", [51, 52, 53, 86, 87, 88, 129, 130, 131])
@pytest.mark.parametrize("c", [1, 3, 4])
def test_rows_of_a_part(pkg, ctx, oracle, h, c):
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize", dict(key="image", w=70, h=20))]
    _check(pkg, ctx, oracle, [(h, 64), (h, 65), (h, 66), (h, 67), (20, 71)], c, ops, seed=h + c)


# along a row: around eleven columns of a strip (2r + 10r + 2 source columns in 241 bytes), and the
# shrinks in between that four channels leave to the other kernel
@pytest.mark.parametrize("c,ratio", [(1, 19.5), (1, 20.5), (2, 9.4), (2, 9.9), (3, 6.3), (3, 6.7), (4, 4.6), (4, 5),
                                     (4, 1.7), (4, 1.8), (4, 3.4), (4, 3.6)])
def test_columns_of_a_strip(pkg, ctx, oracle, c, ratio):
    w = int(12 * ratio)
    ops = [("image_resize", dict(key="image", w=12, h=11)), ("image_random_h_flip", dict(key="image", prob=0.5))]
    _check(pkg, ctx, oracle, [(13, w + k) for k in range(-9, 10, 3)] + [(12, 60)], c, ops, seed=c)


# strips, passes and walks of every remainder: enlargements (many columns a strip) and shrinks
@pytest.mark.parametrize("out", [(1, 1), (3, 31), (4, 32), (5, 33), (127, 65), (129, 256), (130, 257), (513, 40)])
@pytest.mark.parametrize("c", [1, 2, 3, 4])
def test_output_sizes(pkg, ctx, oracle, out, c):
    ops = [("image_resize", dict(key="image", w=out[1], h=out[0]))]
    _check(pkg, ctx, oracle, [(2, 1), (31, 33), (64, 61), (150, 302), (77, 243)], c, ops, seed=out[0],
           casts=(([0.4] * c, [0.2] * c),))


@pytest.mark.parametrize("c", [1, 3])
def test_kernels_mixed_in_ragged_slots(pkg, ctx, oracle, c):
    side = [("image_resize_smallest_side", dict(key="image", size=24))]
    _check(pkg, ctx, oracle, [(24, 30), (200, 40), (40, 900), (700, 720), (50, 61), (24, 24), (31, 500)], c, side, seed=c)


def test_rows_that_start_at_any_byte(pkg, ctx, oracle):
    for cut in range(5):
        ops = [("image_center_crop", dict(key="image", w=100 + cut, h=60)), ("image_resize", dict(key="image", w=90, h=44))]
        _check(pkg, ctx, oracle, [(70, 120 + k) for k in range(6)], 3, ops, seed=cut, casts=(None,))


# which lane takes which column: an enlargement's stay in order, a shrink's are dealt
@pytest.mark.parametrize("c", [1, 2, 3, 4])
def test_order_of_columns(pkg, ctx, oracle, c):
    ops = [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize", dict(key="image", w=70, h=21))]
    _check(pkg, ctx, oracle, [(20, w) for w in (1, 5, 34, 35, 36, 69, 70, 71, 72, 141)], c, ops, seed=c)
