"""Two threads on one context: the ops of one call each, which share a lane, and a lane that one
thread queues on while the other waits for it.  No call of them fails, and every byte is the
oracle's."""
import ctypes
import threading

import numpy as np
import pytest

import chain

pytestmark = pytest.mark.gpu


def _run(*bodies):
    failed = []

    def guarded(body):
        try:
            body()
        except BaseException as e:   # (what a thread raises would be lost)
            failed.append(e)

    threads = [threading.Thread(target=guarded, args=(b,)) for b in bodies]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]


def test_ops_of_two_threads(pkg, oracle):
    own = pkg.Context(device=0, n_lanes=1)
    img = np.random.default_rng(0).integers(0, 256, (61, 47, 3), dtype=np.uint8)
    m = (0.8, -0.6, 1.5, 0.6, 0.8, -2.0)
    i64 = ctypes.c_int64
    turned = np.empty((50, 40, 3), np.uint8)
    oracle.lib().oracle_affine(oracle._p8(img), i64(61), i64(47), i64(3), (ctypes.c_float * 6)(*m), i64(50), i64(40),
                               oracle._p8(turned))
    resized = oracle.resize(img, 30, 20)

    def resizes():
        for _ in range(400):
            assert np.array_equal(own.image_resize(img, 30, 20), resized)

    def rotations():
        for _ in range(400):
            assert np.array_equal(own.image_affine(img, m, 50, 40), turned)

    try:
        _run(resizes, rotations)
    finally:
        own.close()


def test_queueing_on_a_lane_that_another_thread_waits_for(pkg, oracle):
    own = pkg.Context(device=0, n_lanes=1)
    rng = np.random.default_rng(1)
    ops = [("image_resize", dict(key="image", w=48, h=40))]
    imgs = [rng.integers(0, 256, (60 + 5 * i, 90, 3), dtype=np.uint8) for i in range(4)]
    descs, outs = [], [np.zeros((1, 40, 48, 3), np.uint8) for _ in range(4)]
    for a in imgs:
        d = np.zeros(1, pkg.SAMPLE_DTYPE)
        chain.fill_descs(d, 0, chain.reduce_chain(a.shape, ops), a.ctypes.data)
        descs.append(d)
    bds = [pkg.make_batch_desc(o, 40, 48, 3, out_dtype=pkg._capi.U8, divisor=1.0) for o in outs]
    done = threading.Event()

    def queues():
        try:
            for i in range(400):
                own.fused_batch(0, descs[i % 4], bds[i % 4])
        finally:
            done.set()

    def waits():
        while not done.is_set():
            own.wait(0)
        own.wait(0)

    try:
        _run(queues, waits)
        for a, o in zip(imgs, outs):
            assert np.array_equal(o[0], oracle.resize(a, 48, 40))
    finally:
        own.close()
