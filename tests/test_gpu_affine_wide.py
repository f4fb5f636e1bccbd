"""Rotations out of sources at the limits of the row-wise path (affine.cu: affine_rows_take): sides
of 2^23 - 1, the last that it takes, and 2^23, and windows of just below 2^31 bytes and of that size or more,
which go pixel by pixel.  All channel counts, the channel reduction, bytes and both casts, mirrors on both
sides, padded slots."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu

CASTS = [None, (), ([0.4, 0.5, 0.6, 0.7], [0.2, 0.3, 0.25, 0.5])]


def _run(pkg, ctx, fields, src, slot_h, slot_w, c, cast, pad):
    """The batch of these samples, which share a source in GPU memory, as numpy."""
    import torch
    capi = pkg._capi
    descs = np.zeros(len(fields), pkg.SAMPLE_DTYPE)
    for i, f in enumerate(fields):
        chain.fill_descs(descs, i, f, src.data_ptr())
    gray = fields[0]["gray"]
    co = 1 if gray else c
    out = torch.full((len(fields), slot_h, slot_w, co), 99, dtype=torch.uint8 if cast is None else torch.float32, device="cuda")
    mean, std = (list(v[:co]) for v in cast) if cast else (None, None)
    bd = pkg.make_batch_desc(out.data_ptr(), slot_h, slot_w, c, out_dtype=capi.U8 if cast is None else capi.F32,
                             divisor=1.0 if cast is None else 255.0, mean=mean, std=std, pad_value=pad, gray=gray,
                             src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
    ctx.fused_batch_on_stream(torch.cuda.current_stream().cuda_stream, descs, bd)
    return out.cpu().numpy()


def _slots(bytes_of, slot_h, slot_w, cast, pad):
    want = np.full((len(bytes_of), slot_h, slot_w, bytes_of[0].shape[2]), pad, np.uint8)
    for i, b in enumerate(bytes_of):
        want[i, :b.shape[0], :b.shape[1]] = b
    if cast is None:
        return want
    want = want.astype(np.float32) / np.float32(255)
    co = want.shape[3]
    return (want - np.float32(cast[0][:co])) / np.float32(cast[1][:co]) if cast else want


@pytest.fixture(scope="module")
def noise():
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    return torch.randint(0, 256, ((1 << 31) + (1 << 17),), dtype=torch.uint8, device="cuda", generator=gen)


@pytest.mark.parametrize("w", [(1 << 23) - 1, 1 << 23])
@pytest.mark.parametrize("c", [1, 2, 3, 4, "gray"])
def test_sides(pkg, ctx, noise, w, c):
    gray = chain.gray_fixed("default") if c == "gray" else None
    c = 3 if gray else c
    img = noise[:3 * w * c].cpu().numpy().reshape(3, w, c)
    fields = []
    for m2, pre_flip, post_flip in ((-2.0 ** 22, 0, 0), (0.25, 0, 1), (2.0 ** 22 - 40, 1, 0), (-2.0 ** 22, 1, 1), (2.0 ** 22 - 9, 0, 1)):
        fields.append(dict(src_h=3, src_w=w, pre_x=0, pre_y=0, pre_w=w, pre_h=3, pre_flip=pre_flip, geom=2, geom_w=70, geom_h=19,
                           mx=[0.96, 0.13, m2, -0.002, 0.2, 0.1], post_x=3, post_y=1, post_w=60, post_h=17,
                           post_flip=post_flip, gray=gray))
    pixels = [chain.interpret(f, img) for f in fields]
    assert all(p.any() for p in pixels)
    for cast in CASTS:
        got = _run(pkg, ctx, fields, noise, 20, 67, c, cast, 7.0)
        assert np.array_equal(got, _slots(pixels, 20, 67, cast, 7))


# the definition's coordinates are exact for whole translations
@pytest.mark.parametrize("h,w,c", [(65535, 32768, 1), (65536, 32768, 1), (65535, 16384, 2), (65536, 16384, 2), (32768, 21845, 3),
                                   (32769, 21845, 3), (65535, 8192, 4), (65536, 8192, 4)])
def test_bytes(pkg, ctx, noise, h, w, c):
    img = noise[:h * w * c].view(h, w, c)
    th, tw = 40, 50
    fields, pixels = [], []
    for dx in (-(w // 2) + 20, w // 2 - 30):
        for dy in (-(h // 2) + 11, h // 2 - 13):
            for flip in (0, 1):
                fields.append(dict(src_h=h, src_w=w, pre_x=0, pre_y=0, pre_w=w, pre_h=h, pre_flip=flip, geom=2, geom_w=tw,
                                   geom_h=th, mx=[1, 0, dx, 0, 1, dy], post_x=0, post_y=0, post_w=tw, post_h=th, post_flip=0,
                                   gray=None))
                ax = np.trunc(np.arange(tw) - tw / 2 + dx + 0.5 + w / 2).astype(np.int64)
                ay = np.trunc(np.arange(th) - th / 2 + dy + 0.5 + h / 2).astype(np.int64)
                inside = ((ay >= 0) & (ay < h))[:, None] & ((ax >= 0) & (ax < w))[None]
                assert inside.any() and not inside.all()
                ay, ax = ay.clip(0, h - 1), ax.clip(0, w - 1)
                ax = w - 1 - ax if flip else ax
                rows = img[int(ay[0]):int(ay[-1]) + 1].cpu().numpy()
                pixels.append(np.where(inside[..., None], rows[ay - ay[0]][:, ax], 0).astype(np.uint8))
    for cast in CASTS:
        assert np.array_equal(_run(pkg, ctx, fields, noise, th, tw, c, cast, 0.0), _slots(pixels, th, tw, cast, 0))
