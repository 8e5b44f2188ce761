"""Launches whose dynamic shared memory depends on the call: a kernel's limit belongs to the process, so calls
of several sizes from several threads, or captured in one graph, must not lower it for one another."""
import ctypes as C
import threading

import numpy as np
import pytest

from fdt_b200 import synth
from fdt_b200.abi import Options

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _voxels(ndir, nvox, nfibres, model=1):
    bvecs = synth.fibonacci_sphere(ndir).astype(np.float32)
    bvals = ((np.arange(ndir) % 4) * 1000.0).astype(np.float32)
    y, _ = synth.make_volume(nvox, synth.Protocol(bvecs, bvals), nfibres, model == 2, 25.0, seed=ndir)
    return y, bvecs, bvals


def _on_threads(torch, calls, repeats):
    """Runs every call (a function of the thread's stream) `repeats` times on a thread, handle and stream of
    its own, all threads at once; returns the status codes that were not 0."""
    from fdt_b200 import lib

    handles = [lib.Handle() for _ in calls]
    barrier, bad = threading.Barrier(len(calls)), []

    def worker(i):
        s = torch.cuda.Stream()
        with handles[i]:
            barrier.wait()
            for _ in range(repeats):
                rc = calls[i](C.c_void_p(s.cuda_stream))
                if rc != 0:
                    bad.append((i, rc))
        s.synchronize()

    th = [threading.Thread(target=worker, args=(i,)) for i in range(len(calls))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for h in handles:
        h.close()
    return bad


def test_fits_of_several_sizes_on_several_threads(torch):
    """Three fibres need more than 48 KB from 370 measurements on, 49 KB at 380 and 63 KB at 512.  The
    calls of voxels that are not finite end at once, so that their launches follow closely."""
    from fdt_b200 import lib

    L, o = lib.load(), Options.make(model=1, nfibres=3)
    fast, whole, results, keep = [], [], [], []
    for ndir in (380, 512, 440, 512):
        y, bvecs, bvals = _voxels(ndir, 2, 3)
        d, nan, bv, bl = (lib.to_device(a) for a in (y, np.full_like(y, np.nan), bvecs, bvals))
        want = lib.fit(o, d, bv, bl)
        got = tuple(torch.zeros_like(w) for w in want)
        keep.append((d, nan, bv, bl))
        results.append((got, want))
        for calls, data in ((fast, nan), (whole, d)):
            vol = lib.make_volume(data, bv, bl)
            calls.append(lambda s, vol=vol, got=got: L.bpx_fit_dev(C.byref(o), C.byref(vol),
                                                                   *(g.data_ptr() for g in got), s))
    torch.cuda.synchronize()
    assert not _on_threads(torch, fast, 3000)
    assert not _on_threads(torch, whole, 50)
    for got, want in results:
        for g, w in zip(got, want):
            assert torch.equal(g.view(torch.int32), w.view(torch.int32))


def test_chains_with_and_without_a_b_matrix_per_voxel_on_several_threads(torch):
    """512 measurements of three fibres: 60 KB with one b-matrix for all voxels, 84 KB with one for each."""
    from fdt_b200 import lib

    L, ndir, n = lib.load(), 512, 3
    y, bvecs, bvals = _voxels(ndir, n, 3)
    d = lib.to_device(y)
    tables = {0: (bvecs, bvals), 1: (np.tile(bvecs, (n, 1, 1)), np.tile(bvals, (n, 1)))}
    calls, results, keep = [], [], []
    for each in (0, 1, 0, 1):
        o = Options.make(model=1, nfibres=3, gradnonlin=each, nburn=0, njumps=2, sampleevery=2)
        bv, bl = (lib.to_device(a) for a in tables[each])
        params, _, _ = lib.fit(o, d, bv, bl)
        want = lib.mcmc(o, d, bv, bl, params)
        got, vol = torch.zeros_like(want), lib.make_volume(d, bv, bl)
        keep.append((o, bv, bl, params, vol))
        results.append((got, want))
        calls.append(lambda s, o=o, vol=vol, params=params, got=got: L.bpx_mcmc_dev(
            C.byref(o), C.byref(vol), params.data_ptr(), None, got.data_ptr(), None, s))
    torch.cuda.synchronize()
    assert not _on_threads(torch, calls, 3000)
    for got, want in results:
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))


def test_batch_of_several_sizes(torch):
    """The largest size is captured first, the smaller one after it."""
    from fdt_b200 import lib

    o = Options.make(f0=1, ardf0=1, nburn=20, njumps=40, sampleevery=10)
    items = []
    for ndir in (512, 380):
        y, bvecs, bvals = _voxels(ndir, 37, 3)
        d, bv, bl = (lib.to_device(a) for a in (y, bvecs, bvals))
        items.append(dict(data=d, bvecs=bv, bvals=bl, model=1, nfibres=3))
    batch = lib.Batch(o, items, autotune=False)
    assert len(batch.buckets()) == 2
    o.model, o.nfibres = 1, 3
    want = [lib.xfibres_dev(o, it["data"], it["bvecs"], it["bvals"]) for it in items]
    for _ in range(2):
        outs = batch.run()
        torch.cuda.synchronize()
        for out, w in zip(outs, want):
            for k in ("th", "ph", "f", "mean_d", "mean_S0", "mean_f", "status"):
                assert torch.equal(out[k].view(torch.int32), w[k].view(torch.int32)), k
    batch.close()
