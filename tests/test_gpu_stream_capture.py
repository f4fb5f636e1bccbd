"""mlxd_fused_batch_on_stream under stream capture: the graph owns the tables of the
call, so it can be replayed between (and after) any number of other calls, and those
go on as if nothing had been captured.  Calls on either side of 512 samples, where
the table of an ordinary call changes the memory it is copied from."""
import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu

OPS = [("image_resize", dict(key="image", w=24, h=20))]


class _Batch:
    def __init__(self, pkg, oracle, n, f32, seed):
        torch = pytest.importorskip("torch")
        capi = pkg._capi
        rng = np.random.default_rng(seed)
        self.imgs = [rng.integers(0, 256, (30 + i % 5, 40 + i % 7, 3), dtype=np.uint8) for i in range(n)]
        self.src = [torch.from_numpy(a).cuda() for a in self.imgs]
        self.descs = np.zeros(n, pkg.SAMPLE_DTYPE)
        for i, (a, t) in enumerate(zip(self.imgs, self.src)):
            chain.fill_descs(self.descs, i, chain.reduce_chain(a.shape, OPS), t.data_ptr())
        self.out = torch.zeros((n, 20, 24, 3), dtype=torch.float32 if f32 else torch.uint8, device="cuda")
        kw = dict(src_mem=capi.MEM_DEVICE, dst_mem=capi.MEM_DEVICE)
        if f32:
            kw.update(mean=[0.125 * seed] * 3, std=[0.5] * 3)
            self.bd = pkg.make_batch_desc(self.out.data_ptr(), 20, 24, 3, **kw)
        else:
            self.bd = pkg.make_batch_desc(self.out.data_ptr(), 20, 24, 3, out_dtype=capi.U8, divisor=1.0, **kw)
        self.oracle, self.f32, self.seed = oracle, f32, seed

    def same(self):
        want = np.stack([self.oracle.resize(t.cpu().numpy(), 24, 20) for t in self.src])
        if self.f32:
            want = (want.astype(np.float32) / np.float32(255) - np.float32(0.125 * self.seed)) / np.float32(0.5)
        got = self.out.cpu().numpy()
        self.out.zero_()
        return np.array_equal(got, want)


@pytest.mark.parametrize("n", [1, 33, 512, 513, 700])
@pytest.mark.parametrize("f32", [False, True])
def test_replays_between_other_calls(pkg, oracle, n, f32):
    torch = pytest.importorskip("torch")
    own = pkg.Context(device=0, n_lanes=1)
    stream = torch.cuda.Stream()
    try:
        with torch.cuda.stream(stream):
            held = _Batch(pkg, oracle, n, f32, 1)
            others = [_Batch(pkg, oracle, k, f32, 2 + i) for i, k in enumerate((n, 3, 600))]
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):   # nothing has run on this context yet
                own.fused_batch_on_stream(stream.cuda_stream, held.descs, held.bd)
            for turn in range(3):
                for o in others:
                    own.fused_batch_on_stream(stream.cuda_stream, o.descs, o.bd)
                graph.replay()
                assert own.stream_status(stream.cuda_stream) == 0
                assert held.same() and all(o.same() for o in others)
                for t in held.src:
                    t.copy_(255 - t)     # a replay reads what the sources hold then
            del graph
    finally:
        own.close()
