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


# strong shrinks down the rows and along them, both, neither, a copy, an enlargement: each has its own grid of cells
MIXED = [(57, 64), (6000, 30), (30, 6000), (41, 40), (2500, 2400), (7, 9), (40, 41), (300, 301)]


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("cast", [None, ()])
def test_samples_of_unlike_grids_in_one_batch(pkg, ctx, oracle, c, cast):
    _check(pkg, ctx, oracle, MIXED, c, [("image_resize", dict(key="image", w=40, h=41))], cast=cast)
    # ragged slots, padded beside and below
    side = [("image_resize_smallest_side", dict(key="image", size=9))]
    _check(pkg, ctx, oracle, [(57, 64), (6000, 40), (40, 5000), (9, 30), (300, 301)], c, side, cast=cast)


def test_unlike_grids_cost_about_what_their_samples_cost(pkg, ctx):
    """A batch of many small images, a tall strong shrink and a wide one takes about as long
    as its parts one after the other (0.6 times on a B200), not the product of their grids (10 times)."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    ops = [("image_resize", dict(key="image", w=224, h=224))]
    stream = torch.cuda.current_stream().cuda_stream

    def launch(shapes):
        imgs = [torch.zeros((h, w, 3), dtype=torch.uint8, device="cuda") for h, w in shapes]
        descs = np.zeros(len(imgs), pkg.SAMPLE_DTYPE)
        for i, t in enumerate(imgs):
            chain.fill_descs(descs, i, chain.reduce_chain(tuple(t.shape), ops), t.data_ptr())
        out = torch.empty((len(imgs), 224, 224, 3), dtype=torch.uint8, device="cuda")
        bd = pkg.make_batch_desc(out.data_ptr(), 224, 224, 3, out_dtype=capi.U8, divisor=1.0,
                                 src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.fused_batch_on_stream(stream, descs, bd)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[1:])

    small, tall, wide = [(60, 80)] * 500, [(22400, 60)], [(60, 22400)]
    assert launch(small + tall + wide) < 3 * (launch(small) + launch(tall) + launch(wide))
