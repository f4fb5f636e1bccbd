"""Mirrored crops whose width is no multiple of four: the last group of four
pixels of a row is partly empty, and its empty places index nothing."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 2, 3, 5, 29, 30, 31, 33, 65])
@pytest.mark.parametrize("c", [1, 3, 4])
def test_mirrored_crop_of_any_width(pkg, ctx, oracle, width, c):
    rng = np.random.default_rng(7 * width + c)
    samples = [{"image": rng.integers(0, 256, (40, 80 + i, c), dtype=np.uint8)} for i in range(3)]
    ops = [("image_random_h_flip", dict(key="image", prob=1.0)), ("image_center_crop", dict(key="image", w=width, h=21))]
    for cast in (None, (), ([0.4] * c, [0.2] * c)):
        arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
        oracle.set_state(3)
        want = [b["image"] for b in oracle.run_chain(samples, ops, 3, {"image": 9.0}, arg)]
        oracle.set_state(3)
        got = chain.run_fused(pkg, ctx, samples, "image", ops, 3, cast, 9.0)
        assert len(want) == len(got) and all(np.array_equal(w, g) for w, g in zip(want, got))


@pytest.mark.parametrize("offset", range(4))
@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("op", ["copy", "mirror", "rotate"])
def test_rows_off_a_16_byte_boundary(pkg, ctx, oracle, offset, c, op):
    """Batches that start 0 to 3 floats behind a boundary, rows of every residue; nothing around them is written."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(c)
    ops = {"copy": [], "mirror": [("image_random_h_flip", dict(key="image", prob=1.0))],
           "rotate": [("image_rotate", dict(key="image", angle=20.0, crop=False))]}[op]
    for width in (4, 9, 66, 71):
        img = rng.integers(0, 256, (19, width, c), dtype=np.uint8)
        oracle.set_state(1)
        f = chain.reduce_chain(img.shape, ops)
        want = chain.interpret(f, img).astype(np.float32) / np.float32(255)
        h, w = want.shape[:2]
        src = torch.from_numpy(img).cuda()
        out = torch.full((offset + 2 * h * w * c + 8,), -3.0, device="cuda")
        descs = np.zeros(2, pkg.SAMPLE_DTYPE)
        for i in range(2):
            chain.fill_descs(descs, i, f, src.data_ptr())
        bd = pkg.make_batch_desc(out.data_ptr() + 4 * offset, h, w, c, src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
        ctx.fused_batch_on_stream(stream, descs, bd)
        got = out.cpu().numpy()
        assert (got[:offset] == -3).all() and (got[offset + 2 * h * w * c:] == -3).all()
        body = got[offset:offset + 2 * h * w * c].reshape(2, h, w, c)
        assert np.array_equal(body[0], want) and np.array_equal(body[1], want)


def test_odd_widths_cost_little_more_than_even_ones(pkg, ctx):
    """Mirrored images of 719x1279 against 720x1280: 1.1 times the time on a B200 (2.05 with single-float stores)."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    stream = torch.cuda.current_stream().cuda_stream
    ops = [("image_random_h_flip", dict(key="image", prob=1.0))]

    def launch(h, w):
        img = torch.zeros((64, h, w, 3), dtype=torch.uint8, device="cuda")
        out = torch.empty((64, h, w, 3), device="cuda")
        descs = np.zeros(64, pkg.SAMPLE_DTYPE)
        for i in range(64):
            chain.fill_descs(descs, i, chain.reduce_chain((h, w, 3), ops), img[i].data_ptr())
        bd = pkg.make_batch_desc(out.data_ptr(), h, w, 3, src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.fused_batch_on_stream(stream, descs, bd)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    assert launch(719, 1279) < 1.75 * launch(720, 1280)
