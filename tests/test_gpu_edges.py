"""Edges of the launch shapes and of the rules that choose between forms of a kernel, each against the
oracle, NumPy in 64 bits, or the same call by the other form.

Where two forms of one computation must agree bit for bit (the fits with and without the b-value
table, chains packed or spread over warps, tracking from lists or by a second pass), equality is exact.
"""
import ctypes as C

import numpy as np
import pytest

from fdt_b200 import synth
from fdt_b200.abi import Options, TrackOptions
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _protocol(ndir, distinct):
    """ndir measurements with `distinct` b-values (0 among them) in turn."""
    g = synth.fibonacci_sphere(ndir).astype(np.float32)
    b = (np.arange(ndir) % distinct) * (3000.0 / max(distinct - 1, 1))
    return g, b.astype(np.float32)


@pytest.mark.parametrize("distinct", [4, 31, 32, 33])
@pytest.mark.parametrize("model,nfibres,f0,nonlin", [(1, 1, 0, 0), (1, 3, 1, 0), (1, 2, 0, 1), (2, 2, 1, 0)])
def test_fit_equals_the_fit_with_a_b_matrix_per_voxel(torch, distinct, model, nfibres, f0, nonlin):
    """The first fit tabulates the isotropic signal for up to 32 b-values of a shared protocol and forms it
    per measurement otherwise; the same protocol given per voxel (never tabulated) must fit alike."""
    from fdt_b200 import lib

    ndir, n = 70, 41  # 41 voxels: no multiple of a block's four warps
    bvecs, bvals = _protocol(ndir, distinct)
    y, _ = synth.make_volume(n, synth.Protocol(bvecs, bvals), nfibres, model == 2, 25.0, seed=distinct)
    d = lib.to_device(y)
    kw = dict(model=model, nfibres=nfibres, f0=f0, nonlin=nonlin)
    shared = lib.fit(Options.make(**kw), d, lib.to_device(bvecs), lib.to_device(bvals))
    each = lib.fit(Options.make(gradnonlin=1, **kw), d, lib.to_device(np.tile(bvecs, (n, 1, 1))),
                   lib.to_device(np.tile(bvals, (n, 1))))
    for a, b in zip(shared, each):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("nvox", [1, 3, 5, 700])
@pytest.mark.parametrize("ndir", [7, 33, 512])
def test_fit_of_a_voxel_does_not_depend_on_the_launch(torch, nvox, ndir):
    """Warps take voxels from a counter of the launch: every voxel is fitted, in any volume alike."""
    from fdt_b200 import lib

    bvecs, bvals = _protocol(ndir, min(ndir, 7))
    y, _ = synth.make_volume(nvox, synth.Protocol(bvecs, bvals), 1, False, 30.0, seed=ndir)
    o = Options.make(model=1, nfibres=1, rician=1)
    d, bv, bl = lib.to_device(y), lib.to_device(bvecs), lib.to_device(bvals)
    lib.prepare_data(d)
    whole = lib.fit(o, d, bv, bl)
    assert bool(torch.isfinite(whole[0]).all()) and bool((whole[0][:, 0] > 0).all())
    for v in {0, nvox // 2, nvox - 1}:
        one = lib.fit(o, d[v : v + 1].contiguous(), bv, bl)
        for a, b in zip(whole, one):
            assert torch.equal(a[v : v + 1].contiguous().view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("ndir", [33, 64, 129])
def test_chains_packed_and_spread_are_equal(torch, ndir):
    """Up to one voxel per scheduler a warp runs one voxel, beyond that one per group of lanes."""
    from fdt_b200 import lib

    limit = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    n = limit + 1
    prot = synth.truncated_three_shell(ndir)
    y, _ = synth.make_volume(n, prot, 2, True, 25.0, seed=ndir)
    o = Options.make(model=2, nfibres=2, rician=1, f0=1, nburn=10, njumps=40, sampleevery=10)
    d, bv, bl = lib.to_device(y), lib.to_device(prot.bvecs), lib.to_device(prot.bvals)
    lib.prepare_data(d)
    params, tau, _ = lib.fit(o, d, bv, bl)
    packed = lib.mcmc(o, d, bv, bl, params, tau)
    for m in (1, limit):
        spread = lib.mcmc(o, d[:m].contiguous(), bv, bl, params[:m].contiguous(), tau[:m].contiguous())
        assert torch.equal(spread.view(torch.int32), packed[:, :, :m].contiguous().view(torch.int32))


@pytest.mark.parametrize("K", [1, 2, 3])
@pytest.mark.parametrize("nvox,ns", [(1, 1), (31, 7), (32, 8), (33, 9), (500, 50)])
def test_finish_and_maps_match_numpy(torch, K, nvox, ns):
    """Means within FP32 rounding (1e-6 relative) of the FP64 means; dyads within 1e-5 of the FP64 principal
    eigenvector up to the FP32 sines and cosines of the samples (1e-6 each over a spread of directions)."""
    from fdt_b200 import lib

    rng = np.random.default_rng(100 * K + ns)
    r = rng.uniform(0.1, 1.0, (6 + 3 * K, ns, nvox)).astype(np.float32)
    for k in range(K):
        centre = rng.uniform(0.3, 2.8, (1, nvox)), rng.uniform(-3.0, 3.0, (1, nvox))
        for q in range(2):
            r[6 + 3 * k + q] = centre[q] + 0.1 * rng.normal(size=(ns, nvox))
    o = Options.make(model=2, nfibres=K, njumps=25 * ns)
    out = lib.finish(o, lib.to_device(r))
    post = {k: v.cpu().numpy() for k, v in lib.postproc(o, out).items()}
    out = {k: v.cpu().numpy() for k, v in out.items()}
    x = r.astype(np.float64)
    order = np.argsort(-x[8::3].sum(1), axis=0, kind="stable")
    for name, row in (("th", 6), ("ph", 7), ("f", 8)):
        assert np.array_equal(out[name], np.take_along_axis(r[row::3], order[:, None, :], 0))
    for name, row in (("mean_d", 0), ("mean_f0", 1), ("mean_tau", 2), ("mean_dstd", 3), ("mean_R", 4), ("mean_S0", 5)):
        assert np.allclose(out[name], x[row].mean(0), rtol=1e-6, atol=0)
    th, ph = out["th"].astype(np.float64), out["ph"].astype(np.float64)
    v = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)])
    w, e = np.linalg.eigh(np.einsum("iksn,jksn->knij", v, v) / ns)
    big = np.take_along_axis(e[..., 2], np.abs(e[..., 2]).argmax(-1)[..., None], -1)
    assert np.allclose(out["dyads"], np.moveaxis(e[..., 2] * np.sign(big), -1, 1), atol=1e-5)
    assert np.allclose(post["dispersion"], 1.0 - w[..., 2], atol=1e-6)
    assert np.allclose(post["mean_th"], th.mean(1), rtol=1e-6, atol=1e-7)
    assert np.allclose(post["mean_ph"], ph.mean(1), rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("nan", [(0,), (1,), (2,), (0, 2), (0, 1, 2)])
def test_finish_with_nan_fractions(torch, nan):
    """A fibre whose fractions hold a NaN compares with no other: position o takes the last fibre with o
    fibres before it, or fibre 0 where there is none."""
    from fdt_b200 import lib

    K, ns, nvox = 3, 9, 40
    rng = np.random.default_rng(len(nan))
    r = rng.uniform(0.1, 1.0, (6 + 3 * K, ns, nvox)).astype(np.float32)
    for k in nan:
        r[8 + 3 * k, 4] = np.nan
    o = Options.make(model=2, nfibres=K, njumps=25 * ns)
    out = {k: v.cpu().numpy() for k, v in lib.finish(o, lib.to_device(r)).items()}
    s = r[8::3].astype(np.float64).sum(1)
    rank = [sum((s[j] > s[i]) | ((s[j] == s[i]) & (j > i)) for j in range(K) if j != i) for i in range(K)]
    for pos in range(K):
        src = np.zeros(nvox, int)
        for i in range(K):
            src[rank[i] == pos] = i
        assert np.allclose(out["mean_f"][pos], s[src, np.arange(nvox)] / ns, rtol=1e-6, atol=0, equal_nan=True)


@pytest.mark.parametrize("a_mn", [0, 1])
@pytest.mark.parametrize("b_mn", [0, 1])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (40, 24, 72), (64, 64, 64), (72, 40, 56), (136, 264, 136), (320, 72, 328)])
def test_gemm_at_the_edges_of_its_spans(torch, M, N, K, a_mn, b_mn):
    """Operand tiles are copied in spans of 64 elements: spans partly and wholly outside the matrix, tiles
    narrower than a span, contractions that end inside one.  FP32 sums of exact BF16 products differ from
    64-bit ones by less than 1e-5 of the sum of magnitudes; the columns next to the matrix stay unread."""
    from fdt_b200 import lib

    g = torch.Generator(device="cpu").manual_seed(M + 3 * N + 7 * K)
    A = torch.randn((M, K), generator=g).to(torch.bfloat16)
    B = torch.randn((N, K), generator=g).to(torch.bfloat16)

    def padded(x):  # rows 8 elements longer than the matrix, NaN past its end
        out = torch.full((x.shape[0], x.shape[1] + 8), float("nan"), dtype=torch.bfloat16, device="cuda")
        out[:, : x.shape[1]] = x.cuda()
        return out

    a, b = padded(A.t() if a_mn else A), padded(B.t() if b_mn else B)
    c = lib.gemm_bf16(a, b, M, N, K, a_mn=bool(a_mn), b_mn=bool(b_mn))
    torch.cuda.synchronize()
    assert lib.poll_error() == 0
    ref = A.double() @ B.double().t()
    bound = 1e-5 * (A.double().abs() @ B.double().abs().t()) + 1e-6
    assert bool(((c.cpu().double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 700])
@pytest.mark.parametrize("ndir", [1, 64, 65, 256, 257, 330, 700])
def test_inference_at_the_edges_of_its_tiles(torch, rows, ndir):
    """All layers run in one launch, 128 rows to a block, the inputs in chunks of 64 of which four are held
    at a time.  Against the NumPy oracle within 1e-2 (activations rounded to BF16 per layer); bit for bit
    the same for any number of rows, and for parameters and outputs at any 4-byte address."""
    import ctypes as C

    from fdt_b200 import learned, lib
    from oracle import mlp_oracle as M

    rng = np.random.default_rng(rows + ndir)
    p = learned.init_params(ndir, 3)
    k, n, _, boff, _ = learned.geometry(ndir)
    for l in range(5):
        p[boff[l]:boff[l] + n[l]] = 0.05 * rng.normal(size=n[l])
    nin = (ndir + 7) // 8 * 8
    x = np.zeros((rows, nin), np.float32)
    x[:, :ndir] = np.exp(-rng.uniform(0.0, 2.0, (rows, ndir)))
    xd = torch.from_numpy(x).to(torch.bfloat16).cuda()
    xq = xd.float().cpu().numpy()

    def run(n, shift):
        pd = torch.zeros(p.size + shift, device="cuda")
        pd[shift:] = torch.from_numpy(p).cuda()
        out = torch.full((n * 32 + shift + 32,), -7.0, device="cuda")
        rc = lib.load().bpx_mlp_forward_dev(ndir, pd.data_ptr() + 4 * shift, n, xd.data_ptr(), out.data_ptr() + 4 * shift,
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        torch.cuda.synchronize()
        assert lib.poll_error() == 0
        assert bool((out[:shift] == -7.0).all()) and bool((out[shift + n * 32:] == -7.0).all())
        return out[shift:shift + n * 32].reshape(n, 32).cpu().numpy()

    out = run(rows, 0)
    ref, _ = M.forward(p, ndir, xq)
    assert np.linalg.norm(out - ref) < 1e-2 * np.linalg.norm(ref)
    assert np.array_equal(out, run(rows, 1))
    assert np.array_equal(out[:(rows + 1) // 2], run((rows + 1) // 2, 0))


@pytest.mark.parametrize("batch", [1, 63, 65, 960, 961, 2049])
def test_gradients_at_the_edges_of_the_batch_split(torch, batch):
    """From 16 chunks of 64 rows (961 rows) the weight gradients' contractions run in two parts.  The bounds
    of the network tests: 2e-2 relative for gradients, 1e-3 for the loss (BF16 activations)."""
    from fdt_b200 import learned, lib
    from oracle import mlp_oracle as M

    ndir = 33
    rng = np.random.default_rng(batch)
    p = learned.init_params(ndir, 3)
    x = np.zeros((batch, learned.nin(ndir)), np.float32)
    x[:, :ndir] = rng.uniform(0.05, 1.2, size=(batch, ndir))
    x = M.bf16(x)
    t = rng.normal(size=(batch, 32)).astype(np.float32)
    tw = rng.uniform(0.0, 1.0, size=(batch, 32)).astype(np.float32)
    pd, xd = torch.from_numpy(p).cuda(), torch.from_numpy(x).to(torch.bfloat16).cuda()
    td, wd = torch.from_numpy(t).cuda(), torch.from_numpy(tw).cuda()
    g, loss = torch.full_like(pd, np.nan), torch.full((1,), np.nan, device="cuda")
    rc = lib.load().bpx_mlp_train_step_dev(ndir, pd.data_ptr(), g.data_ptr(), batch, xd.data_ptr(), td.data_ptr(),
                                           wd.data_ptr(), loss.data_ptr(),
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and lib.poll_error() == 0
    out, cache = M.forward(p, ndir, x)
    lref, dz = M.loss_grad(out, t, tw)
    gref, gg = M.backward(p, ndir, cache, dz), g.cpu().numpy().astype(np.float64)
    assert abs(loss.item() - lref) <= 1e-3 * abs(lref)
    assert np.linalg.norm(gg - gref) <= 2e-2 * np.linalg.norm(gref)


@pytest.mark.parametrize("nparticles", [1, 31, 400])
@pytest.mark.parametrize("kw", [
    dict(),
    dict(ways=1),
    dict(ways=1, targets=1),
    dict(ways=1, targets=1, distthresh=3.0),  # path lengths are needed: tracked twice
    dict(ways=1, pathdist=1, loopcheck=1),
    dict(modeuler=1, steplength=3.7),  # the test jump reaches past the neighbouring voxel
    dict(sampvox=1, randfib=3, targets=1),
], ids=lambda k: "-".join(k) or "plain")
def test_tracking_small_calls_equal_oracle(torch, nparticles, kw):
    """Calls with fewer particles than a launch has threads, on a mask with an isolated voxel and holes (the
    samples of voxels out of the mask's reach are not repacked), by every way of counting kept halves."""
    from fdt_b200 import lib

    kw = dict(kw)
    th, ph, f, mask = synth.fibre_field((37, 12, 9), nsamples=5, seed=4)
    mask[:] = mask * (np.random.default_rng(1).random(mask.shape) > 0.02)
    mask[0, 0, 0] = 1.0
    planes = [np.zeros_like(mask) for _ in range(2)]
    planes[0][:, :, 14], planes[1][:, :, 22] = 1.0, 1.0
    ways = planes if kw.pop("ways", 0) else None
    targets = planes[::-1] if kw.pop("targets", 0) else None
    o = TrackOptions.make(nparticles=nparticles, nsteps=300, seed=9, **kw)
    seeds = np.array([[18, 6, 4], [0, 0, 0], [30, 6, 4]], np.float32)
    got = lib.probtrack(o, *(lib.to_device(q) for q in (th, ph, f, mask)), seeds, waypoints=ways, targets=targets)
    want = O.probtrack(o, th, ph, f, mask, seeds, waypoints=ways, targets=targets)
    assert np.array_equal(got[0].cpu().numpy(), want[0]) and got[1] == want[1]
    if targets is not None:
        assert np.array_equal(got[2], want[2])


@pytest.mark.parametrize("nfibres", [1, 2, 3])
@pytest.mark.parametrize("nsamples", [1, 31, 32, 33, 50])
@pytest.mark.parametrize("shape", [(37, 12, 9), (16, 8, 8)])
def test_tracking_equals_oracle_for_any_sample_count(torch, nfibres, nsamples, shape):
    """The samples are repacked in tiles of 32 voxels by 32 samples, by a kernel per fibre count: counts below,
    at and past whole tiles, with and without a partial tile of voxels; a fibre without a direction."""
    from fdt_b200 import lib

    th, ph, f, mask = synth.fibre_field(shape, nsamples=nsamples, seed=nsamples)
    th, ph, f = (np.ascontiguousarray(np.concatenate([q] * 3)[:nfibres]) for q in (th, ph, f))
    th[-1, :, :, :, ::5] = 0.0
    o = TrackOptions.make(nparticles=200, nsteps=300, seed=3, randfib=1)
    seeds = np.array([[shape[0] // 2, shape[1] // 2, shape[2] // 2]], np.float32)
    got = lib.probtrack(o, *(lib.to_device(q) for q in (th, ph, f, mask)), seeds)
    want = O.probtrack(o, th, ph, f, mask, seeds)
    assert np.array_equal(got[0].cpu().numpy(), want[0]) and got[1] == want[1]
