"""Batches on a caller's stream whose sample records travel with the launch - none, few (24) or
more (128) of them - and those above, read from a table: resizes like and unlike, copies,
rotations, padded slots, shrinks that are always read from a table.  Several calls are queued before the
first is looked at.  Every value against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NORM = ([0.4, 0.5, 0.6], [0.2, 0.3, 0.25])
CHAINS = {
    "resize": [("image_random_h_flip", dict(key="image", prob=0.5)), ("image_resize", dict(key="image", w=37, h=29))],
    "pad": [("image_resize_smallest_side", dict(key="image", size=24))],
    "crop": [("image_random_crop", dict(key="image", w=17, h=13)), ("image_random_h_flip", dict(key="image", prob=0.5))],
    "ragged": [],
    "rotate": [("image_rotate", dict(key="image", angle=21.0, crop=True)), ("image_center_crop", dict(key="image", w=18, h=15))],
    "gray": [("image_resize", dict(key="image", w=20, h=30)), ("image_channel_reduction", dict(key="image", preset="default"))],
    "strong": [("image_resize", dict(key="image", w=3, h=2))],
}


@pytest.mark.parametrize("name", sorted(CHAINS))
@pytest.mark.parametrize("n", [1, 2, 23, 24, 25, 127, 128, 129])
@pytest.mark.parametrize("cast", [None, (), NORM])
def test_batches(pkg, oracle, name, n, cast):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    ops = CHAINS[name]
    shapes = [(int(rng.integers(20, 70)), int(rng.integers(20, 70))) for _ in range(3 * n)]
    if name == "resize" and n > 2:
        shapes[1], shapes[2] = (400, 21), (22, 380)   # tall and wide: samples count their own cells off
    host = [{"image": rng.integers(0, 256, (h, w, 3), dtype=np.uint8)} for h, w in shapes]
    if name == "gray" and cast is NORM:
        cast = ([0.4], [0.2])
    arg = None if cast is None else {"image": None if len(cast) == 0 else tuple(np.array(v, np.float32) for v in cast)}
    oracle.set_state(n)
    want = [b["image"] for b in oracle.run_chain(host, ops, n, {"image": 5.0}, arg)]
    dev = [{"image": torch.from_numpy(s["image"]).cuda()} for s in host]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    pkg.core.set_device_output(True)
    pkg.core.set_stream(stream.cuda_stream, True)
    try:
        ds = pkg.buffer_from_vector(dev)
        for op, kw in ops:
            ds = getattr(ds, op)(**kw)
        ds = ds.batch(n, pad={"image": 5.0})
        if cast is not None:
            ds = ds.key_cast("image", **({} if len(cast) == 0 else dict(mean=list(cast[0]), std=list(cast[1]))))
    finally:
        pkg.core.set_stream(0, False)
        pkg.core.set_device_output(False)
    pkg.core.set_state(n)
    got = [ds[i]["image"] for i in range(3)]
    with torch.cuda.stream(stream):
        got = [torch.as_tensor(b, device="cuda").cpu().numpy() for b in got]
    assert pkg.core.stream_status(stream.cuda_stream) in (0, None)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and np.array_equal(g, w)
