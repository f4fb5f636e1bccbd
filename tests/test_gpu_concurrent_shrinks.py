"""Two host threads that launch resizes of different shared-memory need at the
same time: neither lowers the kernel's limit under the other."""
import threading

import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 3, 4])
def test_two_threads_of_strong_shrinks(pkg, ctx, oracle, c):
    rows = (4, 5)   # from 2000: plans of 57 to 60 KB and of 51 to 54 KB
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    rng = np.random.default_rng(c)
    img = rng.integers(0, 256, (2000, 24, c), dtype=np.uint8)
    dev = torch.from_numpy(img).cuda()
    torch.cuda.synchronize()
    outs = [torch.zeros((1, h, 20, c), dtype=torch.float32, device="cuda") for h in rows]
    torch.cuda.synchronize()
    failed = []
    start = threading.Barrier(2)

    def work(lane):
        h = rows[lane]
        descs = np.zeros(1, pkg.SAMPLE_DTYPE)
        chain.fill_descs(descs, 0, chain.reduce_chain(img.shape, [("image_resize", dict(key="image", w=20, h=h))]),
                         dev.data_ptr())
        bd = pkg.make_batch_desc(outs[lane].data_ptr(), h, 20, c, src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
        start.wait()
        for i in range(3000):
            try:
                ctx.fused_batch(lane, descs, bd)
            except pkg.MlxdError as e:
                failed.append((lane, i, str(e)))
                break
        ctx.wait(lane)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for h, out in zip(rows, outs):
        want = oracle.resize(img, 20, h).astype(np.float32) / np.float32(255)
        assert np.array_equal(out[0].cpu().numpy(), want)


def test_two_threads_of_strips(pkg, ctx, oracle):
    """Batches whose plans take 50.0 and 49.8 KB, more than a kernel may have unasked: the strips'
    limit is one value for all threads as well."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    rng = np.random.default_rng(0)
    tall, small = rng.integers(0, 256, (400, 300, 3), dtype=np.uint8), rng.integers(0, 256, (60, 60, 3), dtype=np.uint8)
    src = {k: torch.from_numpy(a).cuda() for k, a in (("tall", tall), ("small", small))}
    heights = (400, 384)    # of the tall images' window: 83 and 81 steps a walk
    outs, batches = [], []
    for h in heights:
        descs = np.zeros(192, pkg.SAMPLE_DTYPE)
        for i in range(192):
            kind, a, size = ("tall", tall[:h], 160) if i % 2 == 0 else ("small", small, 256)
            ops = [("image_resize", dict(key="image", w=size, h=size))]
            chain.fill_descs(descs, i, chain.reduce_chain(a.shape, ops), src[kind].data_ptr())
        outs.append(torch.zeros((192, 256, 256, 3), dtype=torch.uint8, device="cuda"))
        batches.append((descs, pkg.make_batch_desc(outs[-1].data_ptr(), 256, 256, 3, out_dtype=capi.U8, divisor=1.0,
                                                   src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)))
    torch.cuda.synchronize()
    failed = []
    start = threading.Barrier(2)

    def work(lane):
        start.wait()
        for i in range(1500):
            try:
                ctx.fused_batch(lane, *batches[lane])
            except pkg.MlxdError as e:
                failed.append((lane, i, str(e)))
                break
        ctx.wait(lane)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for h, out in zip(heights, outs):
        got = out.cpu().numpy()
        assert (got[::2, :160, :160] == oracle.resize(tall[:h], 160, 160)).all()
        assert (got[1::2] == oracle.resize(small, 256, 256)).all()
