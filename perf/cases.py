"""The work a user of this package has it do, as cases that can be timed and compared.

Every case goes through the public entry points (``fdt_b200.lib``, ``fdt_b200.learned``).  The kinds:

* ``pipeline``: a volume or subpart through the fits, the chains and the finishing, on device
  buffers (LM-started or network-started) or on host arrays;
* ``batch``: volumes of mixed sizes, protocols, models and fibre counts in one graph launch;
* ``fit``: the initial fits alone (what a caller of ``bpx_fit_dev`` and the label maker run);
* ``finish``: recorded chains to sorted samples, means and dyads, then the post-processing maps;
* ``net_forward`` / ``net_train``: the initialiser network's inference and one training step;
* ``track``: probtrackx on posterior samples, from single seed points to a seed mask.

``listed()`` has one fixed case for each use, ``draw()`` gives further ones over the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fdt_b200 import learned, lib, synth
from fdt_b200.abi import Options, TrackOptions

MAX_PIPELINE_WORK = 12800 * 288  # voxels x measurements of the largest pipeline case


def listed():
    return [
        # the small CPU-runnable configuration: 500 voxels, the latency of one short call
        dict(name="plain_small", kind="pipeline", form="plain", nvox=500, ndir=64, shells=1, model=1, nfibres=2,
             rician=0, f0=0, nburn=1000),
        # one subpart of xfibres_gpu (12800 voxels) at the whole-brain options, LM start: the largest case
        dict(name="plain_subpart", kind="pipeline", form="plain", nvox=12800, ndir=288, shells=3, model=2, nfibres=3,
             rician=1, f0=1, nburn=1000),
        # the same subpart in the learned form (network start and widths, short burn-in)
        dict(name="learned_subpart", kind="pipeline", form="learned", nvox=12800, ndir=288, shells=3, model=2,
             nfibres=3, rician=1, f0=1, nburn=200),
        # the drop-in host entry on a ragged part; b-values as scanners write them (not exactly equal in a shell)
        dict(name="host_ragged", kind="pipeline", form="host", nvox=3001, ndir=129, shells=3, b_jitter=1, model=2,
             nfibres=2, rician=0, f0=0, nburn=1000),
        # many small volumes at once: sizes, measurement counts, models and fibre counts mixed
        dict(name="batch_mixed", kind="batch", nitems=5, nvox=9000, mix=31, nburn=1000),
        # the initial fits of a part at the whole-brain options
        dict(name="fit_whole_brain", kind="fit", nvox=8192, ndir=288, shells=3, model=2, nfibres=3, rician=1, f0=1),
        # the output side of a sub-volume: 65536 voxels x 50 samples
        dict(name="finish_subvolume", kind="finish", nvox=65536, nfibres=3, nsamples=50),
        # network inference over a sub-volume
        dict(name="net_forward", kind="net_forward", rows=65536, ndir=288),
        # one training step (forward, backward, Adam) at the training program's batch size
        dict(name="net_train", kind="net_train", rows=4096, ndir=288),
        # simple mode: a few seed points, one path distribution each
        dict(name="track_points", kind="track", nx=96, ny=96, nz=60, nfibres=2, nsamples=50, nseeds=4, particles=5000,
             per_seed=1, waypoints=0, targets=0, loopcheck=0, distthresh=0),
        # seedmask mode: a mask of seeds on the three-fibre field
        dict(name="track_mask", kind="track", nx=96, ny=96, nz=60, nfibres=3, nsamples=50, nseeds=512, particles=5000,
             per_seed=0, waypoints=0, targets=0, loopcheck=0, distthresh=0),
        # a connectivity run: waypoints, seeds to targets and the loop check on an odd grid
        dict(name="track_connect", kind="track", nx=73, ny=91, nz=55, nfibres=2, nsamples=50, nseeds=101,
             particles=2000, per_seed=0, waypoints=2, targets=3, loopcheck=1, distthresh=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pipeline", "pipeline", "pipeline", "batch", "fit", "finish", "net_forward", "net_train", "track",
                       "track"])
    if kind in ("pipeline", "fit"):
        ndir = _log_int(rng, 33, 400)
        nvox = _log_int(rng, 200, min(12800, MAX_PIPELINE_WORK // ndir))
        ric = rng.randint(0, 1)
        c = dict(kind=kind, nvox=nvox, ndir=ndir, shells=3 if ndir > 80 else rng.choice([1, 3]), b_jitter=rng.randint(0, 1),
                 model=rng.choice([1, 2, 2, 3]), nfibres=rng.randint(1, 3), rician=ric, f0=rng.randint(0, 1))
        if kind == "pipeline":
            c["form"] = rng.choice(["plain", "plain", "learned", "host"])
            c["nburn"] = 200 if c["form"] == "learned" else 1000
        return c
    if kind == "batch":
        return dict(kind=kind, nitems=rng.randint(2, 5), nvox=_log_int(rng, 1000, 9000), mix=rng.randint(0, 1 << 20),
                    nburn=1000)
    if kind == "finish":
        return dict(kind=kind, nvox=_log_int(rng, 500, 65536), nfibres=rng.randint(1, 3), nsamples=rng.choice([10, 25, 50]))
    if kind == "net_forward":
        return dict(kind=kind, rows=_log_int(rng, 200, 65536), ndir=rng.choice([33, 65, 129, 279, 288]))
    if kind == "net_train":
        return dict(kind=kind, rows=_log_int(rng, 512, 8192), ndir=rng.choice([65, 129, 279, 288]))
    nseeds = _log_int(rng, 1, 256)
    return dict(kind=kind, nx=rng.randint(40, 96), ny=rng.randint(40, 96), nz=rng.randint(20, 60),
                nfibres=rng.randint(1, 3), nsamples=rng.choice([20, 50]), nseeds=nseeds,
                particles=_log_int(rng, 500, 5000), per_seed=int(nseeds <= 8), waypoints=rng.choice([0, 0, 1, 3]),
                targets=rng.choice([0, 0, 2]), loopcheck=rng.choice([0, 0, 1]), distthresh=rng.choice([0, 0, 20]))


# ---- inputs ----------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _protocol(ndir, shells, jitter=0):
    """(bvecs [3][ndir], bvals [ndir]): the configurations' protocols, and others of their form."""
    if ndir == 288 and shells == 3:
        p = synth.three_shell(18, 90)
    elif ndir == 64 and shells == 1:
        p = synth.single_shell_64()
    elif shells == 1:
        nb0 = max(1, ndir // 16)
        g = synth.fibonacci_sphere(ndir - nb0)
        p = synth.Protocol(np.concatenate([np.zeros((3, nb0)), g], 1).astype(np.float32),
                           np.concatenate([np.zeros(nb0), np.full(ndir - nb0, 1000.0)]).astype(np.float32))
    elif ndir <= 279:
        p = synth.truncated_three_shell(ndir)
    else:
        per = (ndir - ndir // 20) // 3
        p = synth.three_shell(ndir - 3 * per, per)
    bvecs, bvals = p.bvecs.copy(), p.bvals.copy()
    if jitter:  # b-values in steps of 5 around their shell's
        step = np.random.default_rng(ndir).integers(-2, 3, ndir) * 5.0
        bvals = np.where(bvals > 0, bvals + step, 0.0).astype(np.float32)
    return bvecs, bvals


def _signals(g, nvox, bvecs, bvals, nfibres, gamma, snr=(20.0, 30.0)):
    """Ball-and-stick voxels with Rician noise, [nvox][ndir] float32 on the device (synth.sample_truth's priors)."""
    gv = torch.as_tensor(bvecs, device="cuda", dtype=torch.float64)
    b = torch.as_tensor(bvals, device="cuda", dtype=torch.float64)[None]
    d = 0.5e-3 + 1.5e-3 * _rand(g, nvox, 1)
    f = [0.3 + 0.4 * _rand(g, nvox, 1)]
    f.append(_rand(g, nvox, 1) * torch.clamp(1.0 - f[0], max=0.3))
    f.append(_rand(g, nvox, 1) * torch.clamp(0.99 - f[0] - f[1], max=0.15))
    s = d * (0.1 + 0.4 * _rand(g, nvox, 1))

    def decay(bc):
        return torch.exp(-(d * d / (s * s)) * torch.log1p(s * s / d * bc)) if gamma else torch.exp(-d * bc)

    sig = (1.0 - sum(f[:nfibres])) * decay(b)
    for k in range(nfibres):
        v = torch.randn((nvox, 3), generator=g, device="cuda", dtype=torch.float64)
        v = v / v.norm(dim=1, keepdim=True)
        sig = sig + f[k] * decay(b * (v @ gv) ** 2)
    sigma = 1000.0 / (snr[0] + (snr[1] - snr[0]) * _rand(g, nvox, 1))
    n = torch.randn((2,) + tuple(sig.shape), generator=g, device="cuda", dtype=torch.float64)
    return torch.sqrt((1000.0 * sig + sigma * n[0]) ** 2 + (sigma * n[1]) ** 2).float().contiguous()


def _options(case, **kw):
    return Options.make(model=case["model"], nfibres=case["nfibres"], rician=case["rician"], f0=case["f0"],
                        ardf0=case["f0"], **kw)


def _weights(ndir):
    """The committed initialiser where there is one for the measurement count, else an untrained one."""
    if ndir in (288, 279):
        return learned.load_weights(learned.default_weights_path("whole_brain" if ndir == 288 else "multishell"))[0]
    return learned.init_params(ndir, seed=ndir)


def _network_inputs(g, rows, ndir):
    bvecs, bvals = _protocol(ndir, 3)
    y = _signals(g, rows, bvecs, bvals, 3, True, (10.0, 40.0))
    x = torch.zeros((rows, learned.nin(ndir)), device="cuda", dtype=torch.bfloat16)
    x[:, :ndir] = (y / y[:, torch.as_tensor(bvals <= 50.0, device="cuda")].mean(1, keepdim=True)).to(torch.bfloat16)
    return x


def _batch_items(case):
    """[(voxels, measurements, model, fibres)] of a mixed batch, from the case alone."""
    r = np.random.default_rng(case["mix"])
    share = np.exp(r.uniform(0.0, math.log(20.0), case["nitems"]))
    n = np.maximum(16, (share / share.sum() * case["nvox"]).astype(int))
    return [(int(v), int(r.choice([33, 65, 129, 279])), int(r.integers(1, 3)), int(r.integers(1, 4))) for v in n]


def _prepare_pipeline(case, seed):
    bvecs, bvals = _protocol(case["ndir"], case["shells"], case.get("b_jitter", 0))
    data = _signals(_gen(seed), case["nvox"], bvecs, bvals, case["nfibres"], case["model"] != 1)
    o = _options(case, nburn=case["nburn"])
    s = dict(case=case, opts=o)
    if case["form"] == "host":
        s.update(data=data.cpu().numpy(), bvecs=bvecs, bvals=bvals)
        return s
    s.update(data=data, bvecs=lib.to_device(bvecs), bvals=lib.to_device(bvals), out=lib.alloc_outputs(o, case["nvox"]))
    if case["form"] == "learned":
        s["net"] = lib.to_device(_weights(case["ndir"]))
    return s


def _prepare_fit(case, seed):
    bvecs, bvals = _protocol(case["ndir"], case["shells"], case.get("b_jitter", 0))
    data = _signals(_gen(seed), case["nvox"], bvecs, bvals, case["nfibres"], case["model"] != 1)
    return dict(case=case, opts=_options(case), data=data, bvecs=lib.to_device(bvecs), bvals=lib.to_device(bvals))


def _prepare_batch(case, seed):
    g, items, tables, first = _gen(seed), [], {}, 0
    for nvox, ndir, model, nfibres in _batch_items(case):
        if ndir not in tables:
            p = synth.truncated_three_shell(ndir)
            tables[ndir] = (p.bvecs, p.bvals, lib.to_device(p.bvecs), lib.to_device(p.bvals))
        bvecs, bvals, dv, dl = tables[ndir]
        items.append(dict(data=_signals(g, nvox, bvecs, bvals, nfibres, model == 2, (10.0, 40.0)), bvecs=dv, bvals=dl,
                          model=model, nfibres=nfibres, voxel_offset=first))
        first += nvox
    return dict(case=case, batch=lib.Batch(Options.make(rician=1, f0=1, ardf0=1, nburn=case["nburn"]), items,
                                           autotune=False))


def _records(case, seed):
    """Chain records [6+3K][nsamples][nvox] (d, f0, tau, d_std, R, S0, then th, ph, f per fibre), as a
    chain leaves them: samples scattered about each voxel's state, angles not wrapped."""
    g, n, ns, K = _gen(seed), case["nvox"], case["nsamples"], case["nfibres"]

    def around(centre, width):
        noise = torch.randn((ns, n), generator=g, device="cuda", dtype=torch.float64)
        return centre[None] + width * noise

    rows = [around(0.5e-3 + 1.5e-3 * _rand(g, n), 3e-5), around(0.05 * _rand(g, n), 1e-3).abs(),
            around(6e-4 + 1e-4 * _rand(g, n), 2e-5), around(4e-4 + 2e-4 * _rand(g, n), 2e-5),
            torch.zeros((ns, n), device="cuda", dtype=torch.float64), around(1000.0 + 20.0 * _rand(g, n), 5.0)]
    for k in range(K):
        th = torch.arccos(2.0 * _rand(g, n) - 1.0) + math.pi * (_rand(g, n) < 0.1)
        ph = 2.0 * math.pi * (_rand(g, n) - 0.5)
        spread = 0.05 * 3.0**k
        rows += [around(th, spread), around(ph, spread),
                 (around((0.7 - 0.3 * k) * _rand(g, n), 0.02)).abs().clamp(max=0.95)]
    return torch.stack(rows).float().contiguous()


def _prepare_train(case, seed):
    g = _gen(seed)
    x = _network_inputs(g, case["rows"], case["ndir"])
    k, n, woff, boff, total = learned.geometry(case["ndir"])
    p = lib.to_device(_weights(case["ndir"]))
    # targets near what the network gives, as later in training; unit weights as the label maker sets
    t = (0.3 * torch.randn((case["rows"], learned.NOUT), generator=g, device="cuda")).float()
    v = t[:, 3:12].reshape(-1, 3, 3)
    t[:, 3:12] = (v / v.norm(dim=2, keepdim=True)).reshape(-1, 9)
    w = torch.rand((case["rows"], learned.NOUT), generator=g, device="cuda")
    # Adam's moments as they stand in the middle of a run
    m = (1e-3 * torch.randn(total, generator=g, device="cuda")).float()
    v2 = (1e-2 * (0.5 + torch.rand(total, generator=g, device="cuda"))) ** 2
    return dict(case=case, x=x, t=t.contiguous(), w=w.contiguous(), p=p, m=m, v=v2.contiguous(), g=torch.zeros_like(p),
                loss=torch.zeros(1, device="cuda"), step=1000)


def _prepare_track(case, seed):
    g = _gen(seed)
    nx, ny, nz, K, ns = (case[k] for k in ("nx", "ny", "nz", "nfibres", "nsamples"))
    z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda", dtype=torch.float32) for n in (nz, ny, nx)), indexing="ij")
    u = [(q - (n - 1) / 2) / (0.48 * n) for q, n in ((x, nx), (y, ny), (z, nz))]
    mask = (u[0] ** 2 + u[1] ** 2 + u[2] ** 2 <= 1.0).float()
    th = torch.empty((K, ns, nz, ny, nx), device="cuda")
    ph, f = torch.empty_like(th), torch.empty_like(th)

    def scatter(width):
        return width * torch.randn((ns, nz, ny, nx), generator=g, device="cuda")

    # a bundle curving along x, one crossing it along y in half the volume, and a weakly supported fibre
    centres = [(math.pi / 2 + 0.3 * u[2], 0.5 * u[0], 0.5 + 0.0 * x), (math.pi / 2 + 0.0 * x, math.pi / 2 + 0.4 * u[1],
               torch.where(x >= nx // 2, 0.3, 0.005)), (1.5 + 0.8 * u[0], 3.0 * u[1], 0.02 + 0.0 * x)]
    for k in range(K):
        th[k], ph[k] = centres[k][0] + scatter(0.08 * 2**k), centres[k][1] + scatter(0.08 * 2**k)
        f[k] = (centres[k][2] + scatter(0.02)).clamp(0.0, 1.0)
    inside = torch.nonzero(mask > 0)
    pick = torch.randint(0, inside.shape[0], (case["nseeds"],), generator=g, device="cuda")
    seeds = inside[pick].flip(1).float().cpu().numpy()
    slabs = [((u[0] + 0.5 - 0.4 * i).abs() < 0.15).float().cpu().numpy() for i in range(3)]
    return dict(case=case, th=th, ph=ph, f=f, mask=mask, seeds=seeds,
                waypoints=slabs[: case["waypoints"]] or None, targets=slabs[: case["targets"]] or None,
                opts=TrackOptions.make(nparticles=case["particles"], per_seed=case["per_seed"],
                                       loopcheck=case["loopcheck"], distthresh=float(case["distthresh"]),
                                       seed=1 + int(seed)))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pipeline":
        return _prepare_pipeline(case, seed)
    if kind == "fit":
        return _prepare_fit(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "finish":
        return dict(case=case, records=_records(case, seed),
                    opts=Options.make(model=2, nfibres=case["nfibres"], rician=1, f0=1, ardf0=1,
                                      njumps=25 * case["nsamples"]))
    if kind == "net_forward":
        return dict(case=case, x=_network_inputs(_gen(seed), case["rows"], case["ndir"]),
                    p=lib.to_device(_weights(case["ndir"])))
    if kind == "net_train":
        return _prepare_train(case, seed)
    return _prepare_track(case, seed)


# ---- one pass --------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pipeline":
        args = (state["opts"], state["data"], state["bvecs"], state["bvals"])
        if case["form"] == "plain":
            return lib.xfibres_dev(*args, out=state["out"])
        if case["form"] == "learned":
            return learned.xfibres_learned(*args, state["net"], freeze=0, out=state["out"])
        return lib.xfibres_host(*args)
    if kind == "fit":
        if case["rician"]:
            lib.prepare_data(state["data"])
        params, tau, status = lib.fit(state["opts"], state["data"], state["bvecs"], state["bvals"])
        return dict(params=params, tau=tau, status=status)
    if kind == "batch":
        return state["batch"].run()
    if kind == "finish":
        out = lib.finish(state["opts"], state["records"])
        post = lib.postproc(state["opts"], out)
        out = {k: v for k, v in out.items() if k != "status"}
        post.update({k: post[k][1:] for k in ("dyads_thr", "dyads_modf")})  # fibre 1's rows are not written
        return dict(out, **post)
    if kind == "net_forward":
        return learned.forward(state["p"], case["ndir"], state["x"])
    if kind == "net_train":
        return _train_step(state)
    r = lib.probtrack(state["opts"], state["th"], state["ph"], state["f"], state["mask"], state["seeds"],
                      waypoints=state["waypoints"], targets=state["targets"])
    return list(r)


def _train_step(s):
    """One mini-batch as learned.train runs it: gradients, then Adam in place."""
    L, ptr, stream = lib.load(), lib._ptr, lib._stream(torch)
    lib._check(L.bpx_mlp_train_step_dev(s["case"]["ndir"], ptr(s["p"]), ptr(s["g"]), s["case"]["rows"], ptr(s["x"]),
                                        ptr(s["t"]), ptr(s["w"]), ptr(s["loss"]), stream), "bpx_mlp_train_step_dev")
    lib._check(L.bpx_mlp_adam_dev(s["p"].numel(), ptr(s["p"]), ptr(s["g"]), ptr(s["m"]), ptr(s["v"]), 1e-4, 0.9, 0.999,
                                  1e-8, s["step"], stream), "bpx_mlp_adam_dev")
    return dict(loss=s["loss"], grads=s["g"], params=s["p"], m=s["m"], v=s["v"])


# ---- what a pass cannot do without -----------------------------------------------------------


def _chain_flops(ndir, model, nfibres, rician, f0, iterations):
    """Per voxel: likelihood evaluations (one per proposal) and the signals each proposal changes."""
    evals = f0 + rician + 1 + (model >= 2) + (model == 3) + 1 + 3 * nfibres
    terms = (nfibres + 1) * ndir * (2 if model == 2 else 1) + (ndir * (1 + nfibres) if model == 3 else 0) + \
        2 * nfibres * ndir
    return iterations * (evals * ndir * 2.0 * (nfibres + 4 + 12 * rician) + terms * 15.0)


def _fit_flops(ndir, model, nfibres, f0):
    """Per voxel: some twenty successful steps of each fit, a model value, a Jacobian row and its outer product each."""
    p = 2 + 3 * nfibres + (model >= 2) + f0
    return (2 if model >= 2 else 1) * 20.0 * ndir * (60.0 * (nfibres + 1) + 2.0 * p * p)


def _output_bytes(nfibres, nsamples):
    return 4.0 * (3 * nfibres * nsamples + 7 + 4 * nfibres + 1)


def work(case):
    kind = case["kind"]
    if kind == "pipeline":
        n, M, K = case["nvox"], case["ndir"], case["nfibres"]
        flops = _chain_flops(M, case["model"], K, case["rician"], case["f0"], case["nburn"] + 1250)
        if case["form"] != "learned":
            flops += _fit_flops(M, case["model"], K, case["f0"])
        return dict(bytes=n * (4.0 * M + _output_bytes(K, 50)), flops=n * flops)
    if kind == "fit":
        n, M, K = case["nvox"], case["ndir"], case["nfibres"]
        return dict(bytes=n * 4.0 * (M + 5 + 3 * K), flops=n * _fit_flops(M, case["model"], K, case["f0"]))
    if kind == "batch":
        b = f = 0.0
        for n, M, model, K in _batch_items(case):
            b += n * (4.0 * M + _output_bytes(K, 50))
            f += n * (_chain_flops(M, model, K, 1, 1, case["nburn"] + 1250) + _fit_flops(M, model, K, 1))
        return dict(bytes=b, flops=f)
    if kind == "finish":
        n, K, ns = case["nvox"], case["nfibres"], case["nsamples"]
        # records in and sorted samples out, the angles in again for the maps, the maps out
        return dict(bytes=n * (4.0 * (6 + 3 * K) * ns + _output_bytes(K, ns) + 8.0 * K * ns + 4.0 * (9 * K + 1)),
                    flops=n * K * ns * 100.0)
    if kind in ("net_forward", "net_train"):
        k, n, _, _, total = learned.geometry(case["ndir"])
        macs = float(sum(a * b for a, b in zip(k, n)))
        rows = case["rows"]
        if kind == "net_forward":
            return dict(bytes=rows * (2.0 * k[0] + 4.0 * learned.NOUT) + 4.0 * total, flops=2.0 * rows * macs)
        # forward, both backward products (none for the inputs), and one update of every parameter
        return dict(bytes=rows * (2.0 * k[0] + 8.0 * learned.NOUT) + 28.0 * total,
                    flops=2.0 * rows * (3.0 * macs - k[0] * n[0]))
    nvox = case["nx"] * case["ny"] * case["nz"]
    # a streamline runs about half the grid's length in steps of half a millimetre (2 mm voxels)
    steps = 2.0 * case["nx"] * case["nseeds"] * case["particles"]
    return dict(bytes=nvox * 12.0 * case["nfibres"] * case["nsamples"] + 4.0 * nvox * (case["nseeds"] if case["per_seed"] else 1),
                flops=steps * 150.0)


# ---- the same in 64 bits ---------------------------------------------------------------------


def exact(case, seed):
    """What run() returns where 64-bit arithmetic gives it (the network and the output side); the
    chains, the fits' stopping points and the integer counts have no such value."""
    if case["kind"] == "finish":
        return _exact_finish(case, seed)
    if case["kind"] == "net_forward":
        s = prepare(case, seed)
        return _network64(s["p"].double(), s["x"].double(), case["ndir"])
    if case["kind"] == "net_train":
        return _exact_train(case, seed)
    return None


def _network64(p, x, ndir):
    k, n, woff, boff, _ = learned.geometry(ndir)
    for l in range(len(k)):
        x = x @ p[woff[l] : woff[l] + n[l] * k[l]].reshape(n[l], k[l]).T + p[boff[l] : boff[l] + n[l]]
        if l + 1 < len(k):
            x = torch.nn.functional.gelu(x)
    return x


def _exact_train(case, seed):
    s = prepare(case, seed)
    p = s["p"].double().requires_grad_(True)
    o, t, w = _network64(p, s["x"].double(), case["ndir"]), s["t"].double(), s["w"].double()
    scalar = [j for j in range(learned.NOUT) if not 3 <= j < 12]
    loss = (w[:, scalar] * (o[:, scalar] - t[:, scalar]) ** 2).sum()
    for k in range(3):
        u, v = o[:, 3 + 3 * k : 6 + 3 * k], t[:, 3 + 3 * k : 6 + 3 * k]
        loss = loss + (w[:, 3 + 3 * k] * ((u * u).sum(1) ** 2 - 2.0 * (u * v).sum(1) ** 2 + 1.0)).sum()
    loss = loss / case["rows"]
    (g,) = torch.autograd.grad(loss, p)
    m = 0.9 * s["m"].double() + 0.1 * g
    v = 0.999 * s["v"].double() + 0.001 * g * g
    new = p.detach() - 1e-4 * (m / (1.0 - 0.9 ** s["step"])) / (torch.sqrt(v / (1.0 - 0.999 ** s["step"])) + 1e-8)
    return dict(loss=loss.detach().reshape(1), grads=g, params=new, m=m, v=v)


def _exact_finish(case, seed):
    r = _records(case, seed).double()
    K, n = case["nfibres"], case["nvox"]
    f = r[8::3]
    order = torch.argsort(f.sum(1), dim=0, descending=True)  # [K][n]
    pick = order[:, None, :].expand(K, r.shape[1], n)
    th, ph, f = (torch.gather(r[6 + q :: 3], 0, pick) for q in range(3))
    v = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)])  # [3][K][ns][n]
    tensor = torch.einsum("iksn,jksn->knij", v, v) / r.shape[1]
    w, e = torch.linalg.eigh(tensor.reshape(-1, 3, 3).cpu())
    w, e = w[:, 2].reshape(K, n).cuda(), e[:, :, 2].reshape(K, n, 3).cuda()
    big = torch.gather(e, 2, e.abs().argmax(2, keepdim=True))
    dyads = torch.where(big < 0, -e, e).permute(0, 2, 1)
    mf = f.mean(1)
    keep = (mf >= 0.05)[:, None].double() * dyads
    return dict(th=th, ph=ph, f=f, mean_d=r[0].mean(0), mean_f0=r[1].mean(0), mean_tau=r[2].mean(0),
                mean_dstd=r[3].mean(0), mean_R=r[4].mean(0), mean_S0=r[5].mean(0), mean_f=mf, dyads=dyads,
                mean_th=th.mean(1), mean_ph=ph.mean(1), dispersion=1.0 - w, dyads_thr=keep[1:],
                dyads_modf=(keep * (mf / mf[0])[:, None])[1:], mean_fsum=mf.sum(0))
