"""Tracking with tables so large that few particles are in flight: kept halves are then tracked twice instead
of being counted from lists, unless a step is short.  Both against the oracle, equal."""
import numpy as np
import pytest

from fdt_b200 import synth
from fdt_b200.abi import TrackOptions
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nparticles", [30, 400], ids=["few", "limited"])
@pytest.mark.parametrize("kw", [
    dict(ways=1),
    dict(avoid=1),
    dict(distthresh=3.0),
    dict(ways=1, targets=1, pathdist=0),
    dict(ways=1, pathdist=1, loopcheck=1),
    dict(ways=1, steplength=0.09),
], ids=lambda k: "-".join(k))
def test_long_paths_equal_oracle(nparticles, kw):
    """2^20 steps: a particle's tables take 32 MB, so seven blocks of 64 particles fit the 16 GB with lists and
    eight without; 90 particles need two of them, 1200 need 19."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fdt_b200 import lib

    kw = dict(kw)
    th, ph, f, mask = synth.fibre_field((37, 12, 9), nsamples=5, seed=4)
    planes = [np.zeros_like(mask) for _ in range(2)]
    planes[0][:, :, 14], planes[1][:, :, 22] = 1.0, 1.0
    ways = planes if kw.pop("ways", 0) else None
    targets = planes[::-1] if kw.pop("targets", 0) else None
    avoid = planes[1] if kw.pop("avoid", 0) else None
    o = TrackOptions.make(nparticles=nparticles, nsteps=1 << 20, seed=9, **kw)
    seeds = np.array([[18, 6, 4], [10, 6, 4], [30, 6, 4]], np.float32)
    got = lib.probtrack(o, *(lib.to_device(q) for q in (th, ph, f, mask)), seeds, waypoints=ways, targets=targets,
                        avoid=None if avoid is None else lib.to_device(avoid))
    want = O.probtrack(o, th, ph, f, mask, seeds, waypoints=ways, targets=targets, avoid=avoid)
    assert np.array_equal(got[0].cpu().numpy(), want[0]) and got[1] == want[1]
    if targets is not None:
        assert np.array_equal(got[2], want[2])
