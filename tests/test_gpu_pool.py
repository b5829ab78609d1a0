"""Reuse of freed device blocks (prad_alloc / prad_free): contents, size classes, recordings, limits."""
import multiprocessing
import threading

import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 4097, 262145])
def test_blocks_are_reused_and_hold_what_is_written_last(n):
    with E.Engine(0) as eng:
        a = np.arange(n, dtype=np.float32)
        for k in range(20):
            m = eng.upload(a + k)
            s = eng.scale(m, 2.0)
            m.free()
            t = eng.scale(s, 0.5)            # may live in m's block
            np.testing.assert_array_equal(t.numpy(), a + k)


def test_a_freed_block_comes_back_and_the_limit_holds():
    with E.Engine(0) as eng:
        m = eng.empty((1000,), np.float32)
        p = m.ptr
        m.free()
        assert eng.empty((1001,), np.float32).ptr == p          # the same size class
        eng.set_option("pool_bytes", "0")
        free0 = eng.device_info()["free_bytes"]
        big = eng.empty((64 << 20,), np.float32)
        big.free()
        assert eng.device_info()["free_bytes"] == free0         # given back at once
        eng.set_option("pool_bytes", str(4 << 30))
        big = eng.empty((64 << 20,), np.float32)
        big.free()
        assert eng.device_info()["free_bytes"] < free0          # kept
        eng.set_option("pool_bytes", "0")
        assert eng.device_info()["free_bytes"] == free0
        with pytest.raises(Exception):
            eng.set_option("pool_bytes", "-1")


def test_blocks_cross_contexts_and_recordings():
    a = np.arange(5000, dtype=np.float64)
    with E.Engine(0) as e1, E.Engine(0) as e2:
        m = e1.upload(a)
        e1.sync()
        E.check(e2.lib.prad_free(e2.ctx, m.ptr))                 # freed by another context
        m.ptr = 0
        x = e1.upload(a)
        seq_out = []
        e1.scale(x, 3.0)
        seq = e1.record(lambda: seq_out.append(e1.scale(x, 3.0)))   # a block born in a recording is not from the cache
        junk = [e1.scale(x, float(k)) for k in range(8)]
        seq.launch()
        np.testing.assert_array_equal(seq_out[0].numpy(), 3.0 * a)
        np.testing.assert_array_equal(junk[5].numpy(), 5.0 * a)
        seq.close()


def test_a_block_is_freed_once():
    a = np.arange(3000, dtype=np.float32)
    with E.Engine(0) as e1, E.Engine(0) as e2:
        m = e1.upload(a)
        p = m.ptr
        m.free()
        for eng in (e1, e2):                                     # the owner again, and another context
            with pytest.raises(E._lib.PradError, match="freed before"):
                E.check(eng.lib.prad_free(eng.ctx, p))
        n = e1.upload(a)                                         # the block is whole, and still given out once
        assert n.ptr == p
        k = e1.upload(a + 1)
        assert k.ptr != p
        np.testing.assert_array_equal(n.numpy(), a)


def _long_work(eng, x, w, y):
    """y = the sum of 40 products of x, some tens of milliseconds; x is read to the end."""
    eng.zero_(y)
    for _ in range(40):
        eng.gemm(x, w, y, beta=1.0)


def _prefetch_into_a_recycled_block(offset):
    n, r = 2048, np.random.default_rng(1)
    with E.Engine(0) as eng:
        a, w = r.standard_normal((n, n)), eng.upload(r.standard_normal((n, n)))
        want, y = eng.empty((n, n), np.float64), eng.empty((n, n), np.float64)
        x = eng.upload(a)
        _long_work(eng, x, w, want)
        want = want.numpy()
        src = eng.pinned_empty((n * n - offset,), np.float64)
        src[:] = r.standard_normal(src.size)
        for _ in range(2):                        # the second time round the copy stream is there
            _long_work(eng, x, w, y)
            p = x.ptr
            x.free()
            new = eng.empty((n, n), np.float64)
            assert new.ptr == p
            part = new.view((n * n - offset,), offset)
            eng.upload_prefetch(src, part)
            eng.upload_join()
            np.testing.assert_array_equal(y.numpy(), want)
            np.testing.assert_array_equal(part.numpy(), src)
            x = new
            eng.upload(a, out=x)
        for m in (x, w, y):
            m.free()


@pytest.mark.parametrize("offset", [0, 4096])
def test_a_prefetch_into_a_recycled_block_waits_for_its_old_work(offset):
    """In a process of its own: with several contexts on the device a recycled block has no old work pending."""
    p = multiprocessing.get_context("spawn").Process(target=_prefetch_into_a_recycled_block, args=(offset,))
    p.start()
    p.join(120)
    assert p.exitcode == 0


def test_a_block_that_another_context_still_reads_is_not_handed_out():
    """The owner frees a matrix that another context's queued work reads, and goes on allocating."""
    n, r = 2048, np.random.default_rng(2)
    a, b = r.standard_normal((n, n)), r.standard_normal((n, n))
    with E.Engine(0) as e1, E.Engine(0) as e2:
        w, y = e2.upload(r.standard_normal((n, n))), e2.empty((n, n), np.float64)
        m = e1.upload(a)
        e1.sync()
        theirs = E.DeviceMatrix(e2, m.ptr, m.shape, m.dtype, owned=False)
        _long_work(e2, theirs, w, y)
        want = y.numpy()
        for _ in range(3):
            _long_work(e2, theirs, w, y)
            m.free()
            m = e1.upload(b)                      # may be the same block
            np.testing.assert_array_equal(y.numpy(), want)
            np.testing.assert_array_equal(m.numpy(), b)
            e1.upload(a, out=m)
            e1.sync()
            theirs.ptr = m.ptr


def test_another_context_may_use_a_new_block_at_once():
    """A block that its owner's queued work still writes is freed, allocated again and given to another context."""
    n, r = 2048, np.random.default_rng(3)
    b = r.standard_normal((n, n))
    with E.Engine(0) as e1:
        x, w = e1.upload(r.standard_normal((n, n))), e1.upload(r.standard_normal((n, n)))
        early = e1.empty((n, n), np.float64)
        _long_work(e1, x, w, early)
        early.free()
        early = e1.empty((n, n), np.float64)      # recycled while the context may be alone
        with E.Engine(0) as e2:
            for new in (early, None, None):
                if new is None:
                    y = e1.empty((n, n), np.float64)
                    _long_work(e1, x, w, y)
                    y.free()
                    new = e1.empty((n, n), np.float64)
                theirs = E.DeviceMatrix(e2, new.ptr, new.shape, new.dtype, owned=False)
                e2.upload(b, out=theirs)
                e2.sync()
                e1.sync()
                np.testing.assert_array_equal(theirs.numpy(), b)
                new.free()


def test_a_packed_operand_dropped_while_recording_is_destroyed_afterwards():
    """As prad_free: its blocks go back to the cache when the recording is closed, and the library refuses to do it before."""
    n, f = 256, np.float32
    a = np.random.default_rng(4).standard_normal((n, n)).astype(f)
    with E.Engine(0) as eng:
        x, out = eng.upload(a), eng.empty((n, n), f)
        ops = [eng.packed(n, n, E.PACK_ROWS | E.PACK_COLS).pack(x)]
        eng.gemm_packed(ops[0], E.PACK_ROWS, ops[0], E.PACK_COLS, out)
        want = out.numpy()

        def step():
            with pytest.raises(E._lib.PradError, match="cannot be recorded"):
                E.check(eng.lib.prad_packed_destroy(ops[0].handle))
            eng.gemm_packed(ops[0], E.PACK_ROWS, ops[0], E.PACK_COLS, out)
            ops.pop().free()
            assert len(eng._deferred_packed) == 1

        eng.zero_(out)
        seq = eng.record(step)
        assert seq.launches >= 1 and not eng._deferred_packed
        assert not out.numpy().any()
        np.testing.assert_allclose(want, a @ a, atol=1e-5 * np.abs(a).max() ** 2 * n)
        seq.close()


def test_threads_with_a_context_each_share_a_matrix():
    """Four threads, a context each, allocate, free and record at the same time; all read matrices of the first thread's context,
    which it frees and replaces while the others' work is queued."""
    n, rounds = 300, 40
    errors = []
    with E.Engine(0) as e0, E.Engine(0) as e1, E.Engine(0) as e2, E.Engine(0) as e3:
        engines = (e0, e1, e2, e3)
        barrier = threading.Barrier(len(engines), timeout=60)
        shared = [None]

        def work(me, eng):
            try:
                r = np.random.default_rng(me)
                for k in range(rounds):
                    if me == 0:
                        shared[0] = e0.upload(np.full((n, n), float(k + 1)))
                        e0.sync()
                    barrier.wait()                # the matrix of this round is there
                    src = E.DeviceMatrix(eng, shared[0].ptr, (n, n), np.float64, owned=False)
                    y = [eng.scale(src, float(f)) for f in range(1, 6)]
                    barrier.wait()                # everybody's work is queued
                    if me == 0:
                        shared[0].free()
                        junk = e0.upload(np.full((n, n), -1.0))
                    a = r.standard_normal(int(r.integers(1, 200000)))
                    m = eng.upload(a)
                    if k % 10 == me:
                        out = eng.empty(a.shape, a.dtype)
                        seq = eng.record(lambda: eng.scale(m, 2.0, out=out))
                        seq.launch()
                        np.testing.assert_array_equal(out.numpy(), 2.0 * a)
                        seq.close()
                    np.testing.assert_array_equal(eng.scale(m, 3.0).numpy(), 3.0 * a)
                    for f, v in enumerate(y, 1):
                        np.testing.assert_array_equal(v.numpy(), np.full((n, n), f * (k + 1.0)))
                        v.free()
                    m.free()
                    if me == 0:
                        junk.free()
            except Exception as ex:               # noqa: BLE001  (the other threads must not wait for this one)
                errors.append((me, repr(ex)))
                barrier.abort()

        threads = [threading.Thread(target=work, args=(i, eng)) for i, eng in enumerate(engines)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(120)
        assert not errors and not any(t.is_alive() for t in threads)
