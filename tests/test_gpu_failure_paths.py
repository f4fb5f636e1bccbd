"""Failure reporting without a fault: a lane wait that runs out of time, and a
resize kernel that finds more source rows than its launch was planned for (a
test hook understates the plan; the CTAs return before they filter anything).
In both cases the caller gets an error code, nothing hangs, and the same context
goes on to produce correct batches."""
import os

import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu

OPS = [("image_resize", dict(key="image", w=48, h=40))]


def _descs(pkg, samples, ops):
    descs = np.zeros(len(samples), pkg.SAMPLE_DTYPE)
    fields = []
    for i, s in enumerate(samples):
        f = chain.reduce_chain(s["image"].shape, ops, s)
        fields.append(f)
        chain.fill_descs(descs, i, f, s["image"].ctypes.data)
    return descs, fields


def test_lane_wait_times_out_and_recovers(pkg, oracle):
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    own = pkg.Context(device=0, n_lanes=1)
    try:
        rng = np.random.default_rng(0)
        # enough work that it cannot be done the moment it is queued
        samples = [{"image": rng.integers(0, 256, (1080, 1920, 3), dtype=np.uint8)} for _ in range(24)]
        ops = [("image_resize_smallest_side", dict(key="image", size=512))]
        descs, fields = _descs(pkg, samples, ops)
        h, w = fields[0]["out_hw"]
        # page-locked destination: the copy back is asynchronous, the call returns with work in flight
        out = torch.zeros((len(samples), h, w, 3), dtype=torch.float32).pin_memory().numpy()
        bd = pkg.make_batch_desc(out, h, w, 3)
        own.fused_batch(0, descs, bd)
        with pytest.raises(pkg.MlxdError) as e:
            own.wait(0, timeout_ms=0)
        assert e.value.code == capi.ERR_TIMEOUT
        own.wait(0)                                   # the work was still queued; now it is done
        want = oracle.resize(samples[0]["image"], w, h).astype("float32") / 255
        d = np.abs(out[0].astype(np.float64) - want.astype(np.float64))
        assert d.max() <= 1.0001 / 255
    finally:
        own.close()


def test_walk_beyond_its_plan_is_reported_and_cleared(pkg, oracle):
    capi = pkg._capi
    own = pkg.Context(device=0, n_lanes=1)
    rng = np.random.default_rng(1)
    samples = [{"image": rng.integers(0, 256, (60, 90, 3), dtype=np.uint8)}]
    descs, fields = _descs(pkg, samples, OPS)
    out = np.zeros((1, 40, 48, 3), np.float32)
    bd = pkg.make_batch_desc(out, 40, 48, 3)
    try:
        os.environ["MLXD_TEST_SHORT_PLAN"] = "1"
        try:
            own.fused_batch(0, descs, bd)
        finally:
            os.environ.pop("MLXD_TEST_SHORT_PLAN", None)
        with pytest.raises(pkg.MlxdError) as e:
            own.wait(0)
        assert e.value.code == capi.ERR_DEVICE and "self-check" in str(e.value)
        # reported once, then cleared: the same lane produces a correct batch
        out[...] = -1
        own.fused_batch(0, descs, bd)
        own.wait(0)
        want = oracle.resize(samples[0]["image"], 48, 40).astype("float32") / 255
        d = np.abs(out[0].astype(np.float64) - want.astype(np.float64))
        assert d.max() <= 1.0001 / 255 and (d > 0).mean() <= 1e-3
    finally:
        own.close()


def test_walk_beyond_its_plan_on_a_stream(pkg, ctx, oracle):
    """The rows that were not filtered keep what the batch held, the padding around them is written."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    stream = torch.cuda.current_stream().cuda_stream
    img = np.random.default_rng(2).integers(0, 256, (200, 90, 3), dtype=np.uint8)
    src = torch.from_numpy(img).cuda()
    descs = np.zeros(1, pkg.SAMPLE_DTYPE)
    chain.fill_descs(descs, 0, chain.reduce_chain(img.shape, OPS), src.data_ptr())
    out = torch.full((1, 50, 300, 3), -1.0, device="cuda")
    bd = pkg.make_batch_desc(out.data_ptr(), 50, 300, 3, pad_value=255.0, src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
    os.environ["MLXD_TEST_SHORT_PLAN"] = "1"
    try:
        ctx.fused_batch_on_stream(stream, descs, bd)
    finally:
        os.environ.pop("MLXD_TEST_SHORT_PLAN", None)
    assert ctx.stream_status(stream) == 8
    assert ctx.stream_status(stream) == 0
    got = out[0].cpu().numpy()
    assert (got[:40, :48] == -1).all() and (got[40:] == 1).all() and (got[:, 48:] == 1).all()
    ctx.fused_batch_on_stream(stream, descs, bd)
    assert ctx.stream_status(stream) == 0
    want = oracle.resize(img, 48, 40).astype(np.float32) / np.float32(255)
    assert np.array_equal(out[0, :40, :48].cpu().numpy(), want)


@pytest.mark.parametrize("h", [200, 1600], ids=["resize_strip", "resize_walk"])
@pytest.mark.parametrize("c", [1, 3, 4])
def test_walk_beyond_its_plan_of_either_kernel(pkg, ctx, oracle, h, c):
    """A shrink by 5 down the rows of two images runs in strips, one by 40 in the kernel of strong
    shrinks: each refuses and recovers."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    stream = torch.cuda.current_stream().cuda_stream
    imgs = [np.random.default_rng(k).integers(0, 256, (h, 90, c), dtype=np.uint8) for k in range(2)]
    src = [torch.from_numpy(a).cuda() for a in imgs]
    descs = np.zeros(2, pkg.SAMPLE_DTYPE)
    for i, (a, t) in enumerate(zip(imgs, src)):
        chain.fill_descs(descs, i, chain.reduce_chain(a.shape, OPS), t.data_ptr())
    out = torch.full((2, 40, 300, c), -1.0, device="cuda")
    bd = pkg.make_batch_desc(out.data_ptr(), 40, 300, c, pad_value=255.0, src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
    os.environ["MLXD_TEST_SHORT_PLAN"] = "1"
    try:
        ctx.fused_batch_on_stream(stream, descs, bd)
    finally:
        os.environ.pop("MLXD_TEST_SHORT_PLAN", None)
    assert ctx.stream_status(stream) == 8
    got = out.cpu().numpy()
    assert (got[:, :, :48] == -1).all() and (got[:, :, 48:] == 1).all()
    ctx.fused_batch_on_stream(stream, descs, bd)
    assert ctx.stream_status(stream) == 0
    for i, a in enumerate(imgs):
        want = oracle.resize(a, 48, 40).astype(np.float32) / np.float32(255)
        assert np.array_equal(out[i, :, :48].cpu().numpy(), want)
