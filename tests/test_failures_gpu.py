"""Failure detection on the GPU without faulting it: a bounded device wait that is made to
run out reports NBODY_ERR_TIMEOUT through the device error word and the context keeps
working; host-side injected failures surface as statuses with reasons, as the reference's
probe / constructor failures do (source/gpu.cpp:115-149, source/sim.cpp:226-239)."""
import ctypes as C
import time

import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu


def test_bounded_wait_times_out_and_the_context_survives(gpu):
    b = golden("disk_512.npz")["bodies"]
    with gpu.Context() as ctx:
        ctx.upload_bodies(b)
        st = gpu.lib().nbody_cuda_selftest_wait(ctx.h, C.c_uint64(1_000_000))     # 1 ms
        assert st == gpu.ERR_TIMEOUT, st
        assert "timed out" in ctx.error()
        # the error word was consumed; the context steps normally afterwards
        ctx.accelerate(gpu.params(law=gpu.LAW_CUTOFF))
        ctx.synchronize()
        acc = ctx.download_bodies()[:, 8:11]
        assert np.isfinite(acc).all() and np.abs(acc).sum() > 0
        assert gpu.lib().nbody_cuda_selftest_wait(ctx.h, C.c_uint64(0)) == gpu.ERR_INVALID


def test_injected_allocation_failure_is_reported(gpu, monkeypatch):
    b = golden("disk_512.npz")["bodies"]
    with gpu.Context() as ctx:
        monkeypatch.setenv("NBODY_CUDA_FAULT", "alloc")
        with pytest.raises(gpu.NbodyError) as e:
            ctx.upload_bodies(b)
        assert e.value.status == gpu.ERR_ALLOC and "injected" in str(e.value)
        monkeypatch.delenv("NBODY_CUDA_FAULT")
        ctx.upload_bodies(b)
        ctx.accelerate(gpu.params(law=gpu.LAW_CUTOFF))
        ctx.synchronize()
    monkeypatch.setenv("NBODY_CUDA_FAULT", "alloc")
    with pytest.raises(gpu.NbodyError) as e:
        gpu.Context()
    assert e.value.status == gpu.ERR_ALLOC


@pytest.mark.parametrize("exported", [False, True])
def test_tree_that_lost_its_buffers(gpu, monkeypatch, exported):
    """A build whose larger buffers cannot be had gives up the last tree's: an export or a query
    of it is then refused, or served from the copy an earlier export left, and never reads the
    buffers that are gone. The next build works again."""
    from nbody_gb300 import scenes
    small, large = scenes.plummer(100, seed=3), scenes.plummer(5000, seed=4)
    p = gpu.params(mode=gpu.MODE_NLOGN, law=gpu.LAW_CUTOFF, theta=0.5, size=0.0, tree_box=1)
    ray = np.array([[0, 0, 0, 1, 2, 3]], np.float32)
    with gpu.Context() as ctx:
        ctx.upload_bodies(small)
        ctx.accelerate(p)
        before = ctx.tree_export() if exported else None
        ctx.upload_bodies(large)
        monkeypatch.setenv("NBODY_CUDA_FAULT", "tree")
        with pytest.raises(gpu.NbodyError) as e:
            ctx.accelerate(p)
        assert e.value.status == gpu.ERR_ALLOC
        monkeypatch.delenv("NBODY_CUDA_FAULT")
        if exported:
            assert np.array_equal(ctx.tree_export(), before)
            assert ctx.tree_query(ray)[1][0] > 0
        else:
            for call in (ctx.tree_export, lambda: ctx.tree_query(ray)):
                with pytest.raises(gpu.NbodyError) as e:
                    call()
                assert e.value.status == gpu.ERR_INVALID
        ctx.accelerate(p)
        nodes = ctx.tree_export()
        assert len(nodes) > 5000 and nodes["mass"][0] == pytest.approx(large[:, 7].sum(dtype=np.float64), rel=1e-6)


def test_look_back_gives_up_as_a_warp(gpu):
    """The self-test makes both bounded waits run out, the second that of the tree build's
    look-back, whose warp votes between its looks: its lanes leave together (the kernel checks
    that), after the limit, and the context goes on to build a tree."""
    from nbody_gb300 import scenes
    with gpu.Context() as ctx:
        ctx.upload_bodies(scenes.plummer(2000, seed=6))
        ctx.synchronize()
        start = time.perf_counter()
        assert gpu.lib().nbody_cuda_selftest_wait(ctx.h, C.c_uint64(50_000_000)) == gpu.ERR_TIMEOUT
        assert time.perf_counter() - start >= 0.1        # 50 ms each
        ctx.accelerate(gpu.params(mode=gpu.MODE_NLOGN, law=gpu.LAW_CUTOFF, theta=0.5, size=0.0, tree_box=1))
        ctx.synchronize()
        assert ctx.bh_stats()["cells"] > 0
