"""Chains of small volumes, one voxel per warp where they are alone on the device and packed where they may run
beside others: the same outputs, and no loss to the others."""
import ctypes as C

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


@pytest.mark.parametrize("ndir", [33, 64, 129, 288])
@pytest.mark.parametrize("over", [-591, 0, 1], ids=["one", "limit", "over"])
def test_pipeline_alone_equals_pipeline_of_a_handle(torch, ndir, over):
    """Unbound pipelines spread up to four voxels per multiprocessor, those of a handle never do."""
    from fdt_b200 import lib

    n = max(1, 4 * torch.cuda.get_device_properties(0).multi_processor_count + over)
    prot = synth.truncated_three_shell(ndir) if ndir < 280 else synth.three_shell(18, 90)
    y, _ = synth.make_volume(n, prot, 2, True, 25.0, seed=ndir)
    o = Options.make(model=2, nfibres=2, rician=1, f0=1, nburn=10, njumps=40, sampleevery=10)
    bv, bl = lib.to_device(prot.bvecs), lib.to_device(prot.bvals)
    alone = lib.xfibres_dev(o, lib.to_device(y), bv, bl)
    h = lib.Handle()
    with h:
        bound = lib.xfibres_dev(o, lib.to_device(y), bv, bl)
    torch.cuda.synchronize()
    h.close()
    for k in alone:
        assert torch.equal(alone[k].view(torch.int32), bound[k].view(torch.int32)), k


def _ms(torch, run):
    best = float("inf")
    for _ in range(4):
        torch.cuda.synchronize()
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        run()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def test_small_chains_beside_one_another_keep_their_speed(torch):
    """Eight times 500 voxels, on streams and as buckets of a batch, against the 4000 at once: the time of
    the packed chains is about the same (spread ones took more than twice as long); the bound is 1.6."""
    from fdt_b200 import lib

    parts, n = 8, 500
    prot = synth.single_shell_64()
    y, _ = synth.make_volume(parts * n, prot, 2, False, 25.0, seed=3)
    d, bv, bl = lib.to_device(y), lib.to_device(prot.bvecs), lib.to_device(prot.bvals)
    o = Options.make(model=1, nfibres=2)
    params, _, _ = lib.fit(o, d, bv, bl)
    main = torch.cuda.current_stream()
    streams = [torch.cuda.Stream() for _ in range(parts)]
    recs = [torch.zeros((lib.nrec(2), o.nsamples, n), device="cuda") for _ in range(parts)]
    whole = torch.zeros((lib.nrec(2), o.nsamples, parts * n), device="cuda")
    volumes = [lib.make_volume(d[i * n : (i + 1) * n], bv, bl, i * n) for i in range(parts)]
    vol, L = lib.make_volume(d, bv, bl), lib.load()

    def at_once():
        assert L.bpx_mcmc_dev(C.byref(o), C.byref(vol), params.data_ptr(), None, whole.data_ptr(), None,
                              C.c_void_p(main.cuda_stream)) == 0

    def on_streams():
        for i, s in enumerate(streams):
            s.wait_stream(main)
            assert L.bpx_mcmc_dev(C.byref(o), C.byref(volumes[i]), params[i * n :].data_ptr(), None, recs[i].data_ptr(),
                                  None, C.c_void_p(s.cuda_stream)) == 0
        for s in streams:
            main.wait_stream(s)

    one, many = _ms(torch, at_once), _ms(torch, on_streams)
    for i in range(parts):
        assert torch.equal(recs[i].view(torch.int32), whole[:, :, i * n : (i + 1) * n].contiguous().view(torch.int32))
    assert many <= 1.6 * one, (many, one)

    def batch(count):  # every copy of the b-vectors makes a bucket of its own
        m = parts * n // count
        items = [dict(data=d[i * m : (i + 1) * m].contiguous(), bvecs=bv.clone(), bvals=bl, model=1, nfibres=2,
                      voxel_offset=i * m) for i in range(count)]
        b = lib.Batch(Options.make(), items, autotune=False)
        assert len(b.buckets()) == count
        t = _ms(torch, b.run)
        b.close()
        return t

    one, many = batch(1), batch(parts)
    assert many <= 1.6 * one, (many, one)
