"""Batches whose sample records are read from a table: their padding and copies cost what those of
batches with the records among the parameters do."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


def test_ragged_copies_from_a_table_cost_little_more(pkg, ctx):
    """256 ragged images in one launch against 128: 1.8 times the time on a B200 (2.4 where each CTA first asked
    for the whole record)."""
    torch = pytest.importorskip("torch")
    capi = pkg._capi
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(2)
    shapes = [(int(h), int(w)) for h, w in rng.integers(200, 401, (128, 2))]
    sources = [torch.zeros((h, w, 1), dtype=torch.uint8, device="cuda") for h, w in shapes]

    def launch(n):
        out = torch.empty((n, 400, 400, 1), dtype=torch.uint8, device="cuda")
        descs = np.zeros(n, pkg.SAMPLE_DTYPE)
        for i in range(n):
            chain.fill_descs(descs, i, chain.reduce_chain((*shapes[i % 128], 1), []), sources[i % 128].data_ptr())
        bd = pkg.make_batch_desc(out.data_ptr(), 400, 400, 1, out_dtype=capi.U8, divisor=1.0, src_mem=capi.MEM_DEVICE,
                                 dst_mem=capi.MEM_DEVICE)
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                ctx.fused_batch_on_stream(stream, descs, bd)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    few, many = launch(128), launch(256)
    print("%.1f us and %.1f, %.2f times" % (few * 50, many * 50, many / few))
    assert many < 2.15 * few
