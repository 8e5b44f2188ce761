"""The fits' launch-wide voxel counter and the largest shared-memory need of the first fit."""
import numpy as np
import pytest

from fdt_b200 import synth
from fdt_b200.abi import Options

pytestmark = pytest.mark.gpu

F0_REFIT = 2  # status bit of a voxel that was fitted again without f0


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _same(torch, got, want):
    return all(torch.equal(g.contiguous().view(torch.int32), w.contiguous().view(torch.int32)) for g, w in zip(got, want))


@pytest.mark.parametrize("model,nfibres", [(2, 3), (1, 2)])
def test_voxels_from_the_counter_equal_voxels_assigned_at_the_start(torch, model, nfibres):
    """The resident warps take their first voxel by their place in the grid and every further one from the
    stage's counter: more than twice as many voxels as warps (20 a multiprocessor), in all four stages, twice
    on one workspace with a smaller volume between, against parts that have a warp for every voxel."""
    from fdt_b200 import lib

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, part = 2 * 20 * sms + 1, 8 * sms
    prot = synth.truncated_three_shell(65)
    y, _ = synth.make_volume(n, prot, nfibres, model == 2, 25.0, seed=model)
    rng = np.random.default_rng(model)
    flat = rng.random(n) < 0.2  # no fibre: their fits take the re-fit stage
    y[flat] = 1000.0 * np.exp(-1e-3 * prot.bvals)[None] + rng.normal(0.0, 40.0, (int(flat.sum()), prot.ndir))
    o = Options.make(model=model, nfibres=nfibres, f0=1, ardf0=1)
    d, bv, bl = lib.to_device(y), lib.to_device(prot.bvecs), lib.to_device(prot.bvals)
    first = lib.fit(o, d, bv, bl)
    lib.fit(o, d[:100].contiguous(), bv, bl)
    again = lib.fit(o, d, bv, bl)
    assert _same(torch, again, first)
    refits = int(((first[2] & F0_REFIT) != 0).sum())
    assert 0 < refits < n
    for v in range(0, n, part):
        few = lib.fit(o, d[v : v + part].contiguous(), bv, bl)
        assert _same(torch, few, [q[v : v + part] for q in first])


@pytest.mark.parametrize("ndir", [369, 370, 512])
@pytest.mark.parametrize("nonlin", [0, 1])
def test_three_fibres_of_many_measurements(torch, ndir, nonlin):
    """Three fibres pass the default limit of 48 KB from 370 measurements on.  The same protocol given per voxel,
    never tabulated, must fit alike."""
    from fdt_b200 import lib

    n = 41
    bvecs = synth.fibonacci_sphere(ndir).astype(np.float32)
    bvals = ((np.arange(ndir) % 4) * 1000.0).astype(np.float32)
    y, _ = synth.make_volume(n, synth.Protocol(bvecs, bvals), 3, False, 25.0, seed=ndir)
    kw = dict(model=1, nfibres=3, f0=1, ardf0=1, nonlin=nonlin)
    d = lib.to_device(y)
    shared = lib.fit(Options.make(**kw), d, lib.to_device(bvecs), lib.to_device(bvals))
    each = lib.fit(Options.make(gradnonlin=1, **kw), d, lib.to_device(np.tile(bvecs, (n, 1, 1))),
                   lib.to_device(np.tile(bvals, (n, 1))))
    assert _same(torch, shared, each)
