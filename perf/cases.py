"""Timed workloads of the XRF path: the calls that reconstruct slices, from one small projection to
whole batches, each with its inputs, its public call and an independent FP64 result.

``listed()`` gives the fixed cases, ``draw(rng)`` another of the same ranges, ``prepare`` what a
program holds before the call, ``run`` one pass of the call, ``work`` the bytes and operations the
call cannot do without, and ``exact`` the same outputs in 64 bits from plain torch.

Inputs are synthetic, with the ranges of the path's data: positive emission images of overlapping
ellipses, linear attenuation of 0 to 0.01 per pixel (scaled with the side), Poisson counts with
peaks of 1e3 to 1e5, angles evenly spaced over a full turn.  Where a case is about projections or
solvers, its attenuation maps are those of a uniform disk, whose line integrals are closed-form;
the map computation has cases of its own.
"""

import ctypes
import math
import os

import numpy as np
import torch

from pycorrectedemissionct_b200 import _lib, core, engine, projectors, solvers, warmstart

EPS32 = float(np.finfo(np.float32).eps)
WEIGHTS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pycorrectedemissionct_b200",
                       "weights", "warmstart.pt")


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one small slice, forward and back: what an interactive script or a per-angle solver calls
        # thousands of times; launches and host work dominate
        dict(name="project_64x48", kind="project", n=64, angles=48, dets=1, dtype="float32"),
        # a slice of awkward size seen by two detectors, maps stored in half the bytes
        dict(name="project_251x361_2det_bf16", kind="project", n=251, angles=361, dets=2, dtype="bfloat16"),
        # the call corrct users make: an MLEM object on one numpy slice with a tolerance
        dict(name="mlem_call_128x180", kind="mlem_call", n=128, angles=180, iterations=40),
        # a batch of slices iterated on the device: the body of every reconstruction
        dict(name="mlem_512x720_16", kind="mlem", n=512, angles=720, slices=16, dtype="float32", iterations=2),
        # the ordered-subsets warm start: one pass over 90 subsets of 8 angles
        dict(name="subsets_512x720_8", kind="subsets", n=512, angles=720, slices=8, subsets=90),
        # attenuation maps of a batch where emitted and incident attenuation are the same volume
        dict(name="maps_512x720_8", kind="maps", n=512, angles=720, slices=8, dets=1, subs=1, same=True,
             dtype="float32"),
        # maps for two finite detectors, an odd number of angles and separate volumes
        dict(name="maps_301x181_2det", kind="maps", n=301, angles=181, slices=2, dets=2, subs=3, same=False,
             dtype="float32"),
        # fluorescence channels of a large slice from shared line integrals, PDHG with TV
        dict(name="pdhg_1024x720_4ch", kind="pdhg", n=1024, angles=720, slices=1, channels=4, iterations=1),
        # a wave of the ragged stream: groups of different sides and angle counts in one launch per
        # operator, SIRT with the attenuated back projection
        dict(name="ragged_sirt_128to512", kind="ragged", n_min=128, n_max=512, angles_min=90, angles_max=360,
             groups=8, slices=2),
        # the exact transpose of the forward projection, for gradients of a user's own data term
        dict(name="adjoint_256x360", kind="adjoint", n=256, angles=360, dets=1),
        # the warm-start network on a batch of slices
        dict(name="net_forward_8x512", kind="net", batch=8, side=512),
        # one convolution layer's gradients at the training batch
        dict(name="conv_backward_16x128_64", kind="conv_backward", batch=16, height=128, width=128, cin=64, cout=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["project", "mlem_call", "mlem", "subsets", "maps", "maps", "pdhg", "ragged", "adjoint", "net",
                       "conv_backward"])
    dtype = rng.choice(["float32", "float32", "bfloat16"])
    if kind == "project":
        return dict(kind=kind, n=_log_int(rng, 32, 512), angles=_log_int(rng, 16, 720), dets=rng.choice([1, 1, 2]),
                    dtype=dtype)
    if kind == "mlem_call":
        return dict(kind=kind, n=_log_int(rng, 48, 256), angles=_log_int(rng, 30, 360), iterations=rng.randint(15, 40))
    if kind == "mlem":
        return dict(kind=kind, n=_log_int(rng, 96, 512), angles=_log_int(rng, 45, 720), slices=_log_int(rng, 1, 12),
                    dtype=dtype, iterations=rng.randint(1, 3))
    if kind == "subsets":
        angles = _log_int(rng, 60, 720)
        return dict(kind=kind, n=_log_int(rng, 96, 512), angles=angles, slices=_log_int(rng, 1, 8),
                    subsets=max(2, angles // rng.choice([8, 8, 12, 40])))
    if kind == "maps":
        same, dets = rng.choice([(True, 1), (False, 1), (False, 2)])
        angles = _log_int(rng, 30, 360)
        return dict(kind=kind, n=_log_int(rng, 64, 512), angles=angles // 4 * 4 if same else angles,
                    slices=_log_int(rng, 1, 4), dets=dets, subs=1 if same else rng.choice([1, 1, 3]), same=same,
                    dtype=dtype)
    if kind == "pdhg":
        return dict(kind=kind, n=_log_int(rng, 128, 768), angles=_log_int(rng, 60, 540), slices=1,
                    channels=rng.randint(2, 4), iterations=rng.randint(1, 3))
    if kind == "ragged":
        n_min, a_min = _log_int(rng, 64, 200), _log_int(rng, 45, 120)
        return dict(kind=kind, n_min=n_min, n_max=_log_int(rng, n_min + 20, 512), angles_min=a_min,
                    angles_max=_log_int(rng, a_min + 10, 360), groups=rng.randint(3, 8), slices=rng.randint(1, 2))
    if kind == "adjoint":
        return dict(kind=kind, n=_log_int(rng, 48, 256), angles=_log_int(rng, 30, 360), dets=rng.choice([1, 1, 2]))
    if kind == "net":
        return dict(kind=kind, batch=rng.randint(1, 8), side=8 * _log_int(rng, 8, 64))
    return dict(kind=kind, batch=rng.randint(2, 16), height=_log_int(rng, 30, 128), width=_log_int(rng, 30, 128),
                cin=rng.choice([16, 32, 64, 128]), cout=rng.choice([16, 32, 64, 128]))


# ----------------------------------------------------------------------------- synthetic inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _angles(a):
    return np.linspace(0.0, 2 * np.pi, a, endpoint=False)


def _ellipses(slices, g, count=12):
    """(S, count, 6): centre x, y, half axes, tilt, value, in units of the half side."""
    u = torch.rand((slices, count, 6), generator=g, device=_dev())
    ax = 0.06 + 0.34 * u[..., :2]
    rad = u[..., 2] * (0.85 - ax.amax(-1))
    ang = 2 * math.pi * u[..., 3]
    return torch.stack([rad * torch.cos(ang), rad * torch.sin(ang), ax[..., 0], ax[..., 1], math.pi * u[..., 4],
                        0.1 + u[..., 5]], -1)


def _image(e, n):
    """Sum of the ellipses on an n x n grid (S, n, n) float32."""
    c = (torch.arange(n, device=_dev(), dtype=torch.float32) - n // 2) / (n / 2)
    y, x = c[None, :, None], c[None, None, :]
    out = torch.zeros((e.shape[0], n, n), device=_dev())
    for k in range(e.shape[1]):
        cx, cy, a, b, psi, v = (e[:, k, i, None, None] for i in range(6))
        p = (x - cx) * torch.cos(psi) + (y - cy) * torch.sin(psi)
        q = (y - cy) * torch.cos(psi) - (x - cx) * torch.sin(psi)
        out += v * ((p / a) ** 2 + (q / b) ** 2 <= 1)
    return out


def _counts(e, n, angles, dets, peak, g):
    """Poisson counts (S, D, A, n) of the ellipses' closed-form projections."""
    s = (torch.arange(n, device=_dev(), dtype=torch.float32) - n // 2) / (n / 2)
    th = torch.as_tensor(np.asarray(angles, dtype=np.float32), device=_dev())
    nx, ny = torch.cos(th)[None, :, None], -torch.sin(th)[None, :, None]
    out = torch.zeros((e.shape[0], len(angles), n), device=_dev())
    for k in range(e.shape[1]):
        cx, cy, a, b, psi, v = (e[:, k, i, None, None] for i in range(6))
        n1 = nx * torch.cos(psi) + ny * torch.sin(psi)
        n2 = ny * torch.cos(psi) - nx * torch.sin(psi)
        w2 = (a * n1) ** 2 + (b * n2) ** 2
        t = s[None, None, :] - (cx * nx + cy * ny)
        out += v * 2 * a * b * torch.sqrt(torch.clamp(w2 - t * t, min=0.0)) / w2
    out = out / out.amax(dim=(1, 2), keepdim=True) * peak
    fade = torch.linspace(1.0, 0.8, dets, device=_dev()) if dets > 1 else torch.ones(1, device=_dev())
    return torch.poisson((out[:, None] * fade[None, :, None, None]).contiguous(), generator=g)


def _disk_maps(slices, n, angles, det_angles, g, dtype="float32", fields=False):
    """Attenuation of a uniform disk per slice, (S, A, D, n, n), or its line integrals
    (S, A, 1 + D, n, n) when ``fields``: path length from each pixel to the rim along the incident
    and the emitted direction, times mu of up to 0.01 per pixel at a side of 512."""
    dev = _dev()
    tdt = torch.bfloat16 if dtype == "bfloat16" else torch.float32
    mu = (0.2 + 0.8 * torch.rand((slices, 1, 1), generator=g, device=dev)) * 0.01 * 512 / n
    rad = (0.30 + 0.12 * torch.rand((slices, 1, 1), generator=g, device=dev)) * n
    c = torch.arange(n, device=dev, dtype=torch.float32) - n // 2
    y, x = c[None, :, None], c[None, None, :]
    r2 = rad * rad - x * x - y * y

    def path(th):
        pd = x * math.sin(th) + y * math.cos(th)
        return mu * torch.clamp(torch.sqrt(torch.clamp(r2 + pd * pd, min=0.0)) - pd, min=0.0)

    planes = len(det_angles) + (1 if fields else 0)
    out = torch.empty((slices, len(angles), planes, n, n), dtype=tdt, device=dev)
    for a, th in enumerate(angles):
        l_in = path(float(th))
        if fields:
            out[:, a, 0] = l_in
        for d, td in enumerate(det_angles):
            l_out = path(float(th) + float(td) + math.pi)
            out[:, a, d + (1 if fields else 0)] = l_out if fields else torch.exp(-l_in - l_out)
    return out


def _mu_disks(slices, n, g, count=5):
    """Linear attenuation (S, n, n): disks of 0 to 0.01 per pixel (at a side of 512), later ones on top."""
    c = (torch.arange(n, device=_dev(), dtype=torch.float32) - (n - 1) / 2) / (n / 2)
    y, x = c[None, :, None], c[None, None, :]
    u = torch.rand((slices, count, 4), generator=g, device=_dev())[..., None, None]
    out = torch.zeros((slices, n, n), device=_dev())
    for k in range(count):
        r = 0.1 + 0.35 * u[:, k, 0]
        rad, ang = u[:, k, 1] * (0.85 - r), 2 * math.pi * u[:, k, 2]
        inside = (x - rad * torch.cos(ang)) ** 2 + (y - rad * torch.sin(ang)) ** 2 <= r * r
        out = torch.where(inside, u[:, k, 3] * 0.01 * 512 / n, out)
    return out.contiguous()


def _det_angles(dets):
    return [math.pi / 2] if dets == 1 else [math.pi / 2, -math.pi / 2][:dets]


def _subset_order(angles, subsets):
    """Every ``subsets``-th angle together: the order of one ordered-subsets level."""
    return np.concatenate([np.arange(r, angles, subsets) for r in range(subsets)])


def _ragged_shapes(case):
    """(n, angles) of the groups, spread over the logarithm of both ranges in opposite orders."""
    g = case["groups"]
    t = [i / max(1, g - 1) for i in range(g)]
    n = [int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** v)) for v in t]
    a = [int(round(case["angles_max"] * (case["angles_min"] / case["angles_max"]) ** v)) for v in t]
    return list(zip(n, a))


def _finite_detectors(case):
    return dict(surfaces_mm2=[25.0] * case["dets"] if case["subs"] > 1 else None,
                distances_mm=[20.0] * case["dets"] if case["subs"] > 1 else None)


def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    kind, g = case["kind"], _gen(seed)
    if kind in ("project", "adjoint"):
        n, a, d = case["n"], case["angles"], case["dets"]
        e = _ellipses(1, g)
        x = _image(e, n)[0].contiguous()
        y = _counts(e, n, _angles(a), d, 1e4, g)[0]
        maps = _disk_maps(1, n, _angles(a), _det_angles(d), g, case.get("dtype", "float32"))
        return dict(x=x, y=y, maps=maps)
    if kind == "mlem_call":
        n, a = case["n"], case["angles"]
        e = _ellipses(1, g)
        return dict(b=_counts(e, n, _angles(a), 1, 1e4, g), maps=_disk_maps(1, n, _angles(a), _det_angles(1), g))
    if kind == "mlem":
        n, a, s = case["n"], case["angles"], case["slices"]
        e = _ellipses(s, g)
        return dict(b=_counts(e, n, _angles(a), 1, 1e5, g),
                    maps=_disk_maps(s, n, _angles(a), _det_angles(1), g, case["dtype"]))
    if kind == "subsets":
        n, s = case["n"], case["slices"]
        ang = _angles(case["angles"])[_subset_order(case["angles"], case["subsets"])]
        e = _ellipses(s, g)
        return dict(angles=ang, b=_counts(e, n, ang, 1, 1e5, g), maps=_disk_maps(s, n, ang, _det_angles(1), g))
    if kind == "maps":
        mu = _mu_disks(case["slices"], case["n"], g)
        return dict(mu_in=mu, mu_out=mu if case["same"] else _mu_disks(case["slices"], case["n"], g))
    if kind == "pdhg":
        n, a, s, c = case["n"], case["angles"], case["slices"], case["channels"]
        e = _ellipses(s * c, g)
        return dict(b=_counts(e, n, _angles(a), 1, 1e3, g), x0=(0.5 + _image(e, n)).contiguous(),
                    scales=np.linspace(0.6, 2.4, c).astype(np.float32),
                    fields=_disk_maps(s, n, _angles(a), _det_angles(1), g, fields=True))
    if kind == "ragged":
        out = []
        for n, a in _ragged_shapes(case):
            e = _ellipses(case["slices"], g)
            out.append(dict(n=n, angles=a, b=_counts(e, n, _angles(a), 1, 1e4, g), x0=_image(e, n).contiguous(),
                            maps=_disk_maps(case["slices"], n, _angles(a), _det_angles(1), g)))
        return dict(groups=out)
    if kind == "net":
        b, h = case["batch"], case["side"]
        planes = []
        for k in range(b):  # 11 increasingly sharp views of one image, as snapshots of an iterate are
            im = _image(_ellipses(1, g), h)
            views = [torch.nn.functional.avg_pool2d(im[None], 2 * (11 - i) + 1, 1, 11 - i)[0] for i in range(11)]
            planes.append(torch.cat(views, 0) / im.mean())
        x = torch.zeros((b, h, h, 16), device=_dev())
        x[..., :11] = torch.stack(planes).permute(0, 2, 3, 1)
        return dict(x=x.to(torch.bfloat16).contiguous())
    if kind == "conv_backward":
        shape = (case["batch"], case["height"], case["width"])
        x = torch.randn((*shape, case["cin"]), generator=g, device=_dev()).relu()
        dy = torch.randn((*shape, case["cout"]), generator=g, device=_dev()) / math.prod(shape)
        w = torch.randn((case["cout"], 9, case["cin"]), generator=g, device=_dev()) * math.sqrt(2 / (9 * case["cin"]))
        return dict(x=x.to(torch.bfloat16), dy=dy.to(torch.bfloat16), w=w.to(torch.bfloat16))
    raise ValueError(f"unknown kind {kind!r}")


# --------------------------------------------------------------------------------- the user's call
def prepare(case, seed):
    kind, t = case["kind"], _inputs(case, seed)
    if kind in ("project", "adjoint"):
        n = case["n"]
        maps = t["maps"][0]
        p = projectors.ProjectorAttenuationXRF(
            (n, n), _angles(case["angles"]), att_maps=maps, angles_detectors_rad=_det_angles(case["dets"]),
            maps_dtype=case.get("dtype", "float32"), bp_mode="adjoint" if kind == "adjoint" else "reference")
        return dict(kind=kind, p=p, x=t["x"], y=t["y"] if case["dets"] > 1 else t["y"][0].contiguous())
    if kind == "mlem_call":
        n = case["n"]
        p = projectors.ProjectorAttenuationXRF((n, n), _angles(case["angles"]), att_maps=t["maps"][0])
        return dict(kind=kind, p=p, b=t["b"][0, 0].cpu().numpy(), iterations=case["iterations"])
    if kind == "mlem":
        c = core.XrfCore(case["n"], _angles(case["angles"]))
        return dict(kind=kind, solver=engine.BatchedSolver(c, t["maps"], t["b"], "mlem"), x0=None,
                    iterations=case["iterations"])
    if kind == "subsets":
        c = core.XrfCore(case["n"], t["angles"])
        return dict(kind=kind, os=engine.OrderedSubsets(c, t["maps"], t["b"], [(case["subsets"], 1)]))
    if kind == "maps":
        args = dict(angles_rad32=np.asarray(_angles(case["angles"]), dtype=np.float32),
                    det_angles=_det_angles(case["dets"]), sub_sampling=case["subs"], maps_dtype=case["dtype"],
                    **_finite_detectors(case))
        return dict(kind=kind, mu_in=t["mu_in"], mu_out=t["mu_out"], args=args)
    if kind == "pdhg":
        c = core.XrfCore(case["n"], _angles(case["angles"]))
        c.set_channels(t["scales"])
        sv = engine.BatchedSolver(c, t["fields"], t["b"], "pdhg", x0=t["x0"], lower_limit=0.0, tv_lambda=1e-2)
        return dict(kind=kind, solver=sv, x0=t["x0"], iterations=case["iterations"])
    if kind == "ragged":
        svs = []
        for gr in t["groups"]:
            c = core.XrfCore(gr["n"], _angles(gr["angles"]))
            svs.append(engine.BatchedSolver(c, gr["maps"], gr["b"], "sirt", x0=gr["x0"], bp_mode="symmetric",
                                            lower_limit=0.0, relaxation=1.0))
        return dict(kind=kind, solvers=svs, ragged=engine.RaggedSolvers(svs))
    if kind == "net":
        net = warmstart.WarmStartNet()
        net.load(WEIGHTS)
        return dict(kind=kind, net=net, x=t["x"])
    if kind == "conv_backward":
        d = _lib.ConvDesc()
        d.batch, d.height, d.width, d.cin, d.cout = (case[k] for k in ("batch", "height", "width", "cin", "cout"))
        back = _lib.ConvDesc()
        back.batch, back.height, back.width, back.cin, back.cout = d.batch, d.height, d.width, d.cout, d.cin
        dev = t["x"].device
        return dict(kind=kind, lib=_lib.load(), desc=d, back=back, **t,
                    wflip=torch.empty((case["cin"], 9, case["cout"]), dtype=torch.bfloat16, device=dev),
                    dw=torch.empty((case["cout"], 9, case["cin"]), device=dev),
                    db=torch.empty(case["cout"], device=dev), dx=torch.empty_like(t["x"]))
    raise ValueError(f"unknown kind {kind!r}")


def run(state):
    kind = state["kind"]
    if kind == "project":
        return state["p"](state["x"]), state["p"].T(state["y"])
    if kind == "adjoint":
        return state["p"].T(state["y"])
    if kind == "mlem_call":
        x, info = solvers.MLEM(tolerance=1e-6)(state["p"], state["b"], iterations=state["iterations"])
        return x, info.residuals.astype(np.float32)
    if kind in ("mlem", "pdhg"):
        sv = state["solver"]
        sv.reset(state["x0"])
        sv.run(state["iterations"], use_graph=False)
        return sv.x if kind == "pdhg" else (sv.x, sv.residuals.float())
    if kind == "subsets":
        return state["os"].run()
    if kind == "maps":
        return core.compute_maps(state["mu_in"], state["mu_out"], **state["args"])
    if kind == "ragged":
        state["ragged"].step()
        return [sv.x for sv in state["solvers"]]
    if kind == "net":
        return state["net"].forward(state["x"])
    # a layer's backward pass: weight, bias and data gradients, through the C interface
    lib, h = state["lib"], core.stream_handle(state["x"].device)
    d, back = ctypes.byref(state["desc"]), ctypes.byref(state["back"])
    x, dy, w, wflip, dw, db, dx = (state[k] for k in ("x", "dy", "w", "wflip", "dw", "db", "dx"))
    dw.zero_()
    db.zero_()
    cin, cout, pixels = state["desc"].cin, state["desc"].cout, dy.numel() // dy.shape[-1]
    _lib.check(lib.cct_conv3x3_wgrad(d, x.data_ptr(), dy.data_ptr(), dw.data_ptr(), h))
    _lib.check(lib.cct_net_bias_grad(dy.data_ptr(), db.data_ptr(), pixels, cout, h))
    _lib.check(lib.cct_net_flip_weights(w.data_ptr(), wflip.data_ptr(), cin, cout, h))
    _lib.check(lib.cct_conv3x3_fwd(back, dy.data_ptr(), wflip.data_ptr(), None, 0, dx.data_ptr(), h))
    return dw, db, dx


# ------------------------------------------------------------------------------ what it cannot save
def work(case):
    """Each input read once and each output written once; one bilinear sample (or lerp) of a
    projection counted with the multiply by its map as 10 (or 4) operations."""
    kind = case["kind"]
    if kind in ("project", "adjoint", "mlem_call", "mlem", "subsets", "pdhg"):
        n, a, d = case["n"], case["angles"], case.get("dets", 1)
        s = case.get("slices", 1) * case.get("channels", 1)
        px, maps, lines = s * n * n, s * a * d * n * n, s * a * d * n
        mb = 2 if case.get("dtype") == "bfloat16" else 4
        if kind == "project":
            return dict(bytes=maps * mb + 8 * px + 8 * lines, flops=14 * maps)
        if kind == "adjoint":
            return dict(bytes=maps * mb + 4 * px + 4 * lines, flops=10 * maps)
        # an iteration: fp (maps, x, b, ratio written), bp (ratio read, x read and written, tau)
        per = dict(bytes=maps * mb + 16 * px + 12 * lines, flops=14 * maps)
        its = case.get("iterations", 1)
        if kind == "subsets":  # x and tau pass once per subset
            per["bytes"] += (case["subsets"] - 1) * 16 * px
        if kind == "pdhg":  # two line-integral planes per angle for all channels; duals and relaxed x
            per["bytes"] = 8 * maps // case["channels"] + 16 * lines + 36 * px
        return dict(bytes=its * per["bytes"], flops=its * per["flops"])
    if kind == "maps":
        n, a, s, d = case["n"], case["angles"], case["slices"], case["dets"]
        out = s * a * d * n * n
        scans = a // 2 if case["same"] else a * (1 + d * case["subs"]) // 2
        return dict(bytes=out * (2 if case["dtype"] == "bfloat16" else 4) + (4 if case["same"] else 8) * s * n * n,
                    flops=2 * 10 * s * scans * n * n)
    if kind == "ragged":
        by = fl = 0
        for n, a in _ragged_shapes(case):
            px, maps, lines = (case["slices"] * v for v in (n * n, a * n * n, a * n))
            by += 8 * maps + 16 * px + 16 * lines  # the maps pass once forward and once back
            fl += 14 * maps
        return dict(bytes=by, flops=fl)
    if kind == "net":
        b, h = case["batch"], case["side"]
        convs = [(16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (64, 128, 4), (128, 128, 4), (128, 256, 8),
                 (256, 256, 8), (256, 128, 4), (128, 128, 4), (128, 64, 2), (64, 64, 2), (64, 32, 1), (32, 32, 1),
                 (32, 16, 1)]
        return dict(bytes=2 * b * h * h * 16 * 2, flops=sum(18 * ci * co * b * (h // q) ** 2 for ci, co, q in convs))
    px = case["batch"] * case["height"] * case["width"]
    ci, co = case["cin"], case["cout"]
    return dict(bytes=2 * px * (2 * ci + co) + (2 + 4) * 9 * ci * co, flops=2 * 18 * ci * co * px)


# --------------------------------------------------------------------------------- FP64, plain torch
def _degrees(angles):
    return np.rad2deg(np.array(angles, ndmin=1, dtype=np.float32))


def _trig(deg):
    r = np.deg2rad(np.asarray([deg], dtype=np.float32))[0]
    return np.cos(r), np.sin(r)


def _bilinear(img, x, y):
    """Bilinear samples of (S, h, w) FP64 images at (x, y), zero outside; (S, *x.shape)."""
    s, h, w = img.shape
    pad = torch.nn.functional.pad(img, (1, 1, 1, 1)).reshape(s, -1)
    fx, fy = torch.floor(x), torch.floor(y)
    dx, dy = (x - fx).reshape(-1), (y - fy).reshape(-1)
    x0, x1 = (torch.clamp(fx + k, -1, w).long().reshape(-1) + 1 for k in (0, 1))
    y0, y1 = ((torch.clamp(fy + k, -1, h).long().reshape(-1) + 1) * (w + 2) for k in (0, 1))
    top = pad[:, y0 + x0] * (1 - dx) + pad[:, y0 + x1] * dx
    bot = pad[:, y1 + x0] * (1 - dx) + pad[:, y1 + x1] * dx
    return (top * (1 - dy) + bot * dy).reshape(s, *x.shape)


def _radon_positions(n, deg):
    c, s = _trig(deg)
    k = n // 2
    m = np.array([c, s, -k * (c + s - 1), -s, c, -k * (c - s - 1)]).astype(np.float64)
    i = torch.arange(n, device=_dev(), dtype=torch.float64)
    return m[0] * i[None, :] + m[1] * i[:, None] + m[2], m[3] * i[None, :] + m[4] * i[:, None] + m[5]


def _fp64(x, map_of, dets, degs):
    """(S, D, A, n) of FP64 images (S, n, n) and map_of(a) -> (S, D, n, n)."""
    s, n = x.shape[0], x.shape[-1]
    out = torch.empty((s, dets, len(degs), n), dtype=torch.float64, device=x.device)
    for a, deg in enumerate(degs):
        z = x[:, None] * map_of(a)
        out[:, :, a] = _bilinear(z.reshape(s * dets, n, n), *_radon_positions(n, deg)).sum(1).reshape(s, dets, n)
    return out


def _lines64(y, n, deg):
    """Back projection of one angle's lines (L, n): (L, n, n)."""
    c, s = (float(v) for v in _trig(deg))
    i = torch.arange(n, device=_dev(), dtype=torch.float64) - n // 2
    u = i[None, :] * c - i[:, None] * s + n // 2
    f = torch.clamp(torch.floor(u), 0, n - 2)
    k = f.long()
    v = y[:, k] + (u - f) * (y[:, k + 1] - y[:, k])
    return torch.where((u >= 0) & (u <= n - 1), v, torch.zeros_like(v))


def _bp64(y, n, degs, map_of=None):
    """(S, n, n) of lines (S, D, A, n), weighted per angle by map_of(a) when given."""
    s, d = y.shape[:2]
    out = torch.zeros((s, n, n), dtype=torch.float64, device=y.device)
    for a, deg in enumerate(degs):
        v = _lines64(y[:, :, a].reshape(s * d, n), n, deg).reshape(s, d, n, n)
        out += (v if map_of is None else v * map_of(a)).sum(1)
    return out


def _adjoint64(y, n, degs, map_of):
    """Exact transpose of ``_fp64`` for one slice: scatter of every bilinear tap."""
    d = y.shape[1]
    out = torch.zeros((n, n), dtype=torch.float64, device=y.device)
    for a, deg in enumerate(degs):
        px, py = _radon_positions(n, deg)
        fx, fy = torch.floor(px), torch.floor(py)
        acc = torch.zeros((d, (n + 2) ** 2), dtype=torch.float64, device=y.device)
        for ky in (0, 1):
            for kx in (0, 1):
                w = (1 - (px - fx - kx).abs()) * (1 - (py - fy - ky).abs())
                tx, ty = torch.clamp(fx + kx, -1, n).long() + 1, torch.clamp(fy + ky, -1, n).long() + 1
                acc.index_add_(1, (ty * (n + 2) + tx).reshape(-1), (w * y[0, :, a][:, None, :]).reshape(d, -1))
        out += (acc.reshape(d, n + 2, n + 2)[:, 1:-1, 1:-1] * map_of(a)[0]).sum(0)
    return out


def _kl64(ax, b):
    r = torch.clamp(ax, min=EPS32)
    return ((1 + r - torch.sqrt((r - 1) ** 2 + 4 * b)) / 2).abs().sum(dim=(1, 2, 3))


def _mlem64(b, n, degs, map_of, iterations, x=None, tau=None):
    b = b.double()
    x = torch.ones((b.shape[0], n, n), dtype=torch.float64, device=b.device) if x is None else x
    tau = _bp64(torch.ones_like(b[:1]), n, degs)
    res = []
    for _ in range(iterations):
        ax = _fp64(x, map_of, b.shape[1], degs)
        res.append(_kl64(ax, b))
        upd = _bp64(b / torch.clamp(ax, min=EPS32), n, degs)
        x = torch.where(tau != 0, x * (upd / tau), x)
    return x, res


def _warp(img, deg, size, sub=None):
    """The images rotated about the centre of their size x size frame, zero outside; ``sub`` crops."""
    r = np.deg2rad(deg)
    c, s, m = math.cos(r), math.sin(r), size / 2.0 - 0.5
    i = torch.arange(size, device=_dev(), dtype=torch.float64)
    i = i if sub is None else i[sub]
    x, y = i[None, :] - m, i[:, None] - m
    return _bilinear(img, c * x - s * y + m, s * x + c * y + m)


def _attenuation64(mu, angle, invert):
    n = mu.shape[-1]
    edge = int(np.ceil((np.ceil(np.sqrt(2.0 * n * n)) - n) / 2))
    size = n + 2 * edge
    if invert:
        angle = angle + np.pi
    deg = np.rad2deg(angle)
    cum = _warp(torch.nn.functional.pad(mu, (edge,) * 4), -deg, size)
    cum = cum + torch.roll(cum, 1, dims=-2)
    cum = torch.cumsum(cum / 2, dim=-2)
    return torch.exp(-_warp(cum, deg, size, slice(edge, edge + n)))


def _maps64(case, t):
    a32 = np.asarray(_angles(case["angles"]), dtype=np.float32)
    subs = np.zeros(1)
    if case["subs"] > 1:
        half = np.arctan2(np.sqrt(25.0) / 2, 20.0)
        edges = np.linspace(-half, half, case["subs"] + 1)
        subs = (edges[:-1] + edges[1:]) / 2
    dets = np.array(_det_angles(case["dets"]))
    mu_in, mu_out = t["mu_in"].double(), t["mu_out"].double()
    s, n = mu_in.shape[0], mu_in.shape[-1]
    out = torch.empty((s, len(a32), len(dets), n, n), dtype=torch.float64, device=mu_in.device)
    for i, a in enumerate(a32):
        f_in = _attenuation64(mu_in, a, False)
        for d, ad in enumerate(a + dets):
            f = sum(_attenuation64(mu_out, ad + v, True) for v in subs) / len(subs)
            out[:, i, d] = f_in * f
    return out


def _pdhg64(case, t):
    n, ch = case["n"], case["channels"]
    degs = _degrees(_angles(case["angles"]))
    b, fields = t["b"].double(), t["fields"]
    sc = torch.as_tensor(t["scales"], device=b.device).double()[None, :, None, None]

    def map_of(a):
        l_in, l_out = fields[:, a, 0].double(), fields[:, a, 1].double()
        return torch.exp(-(l_in[:, None] + sc * l_out[:, None])).reshape(-1, 1, n, n)

    x = t["x0"].double()
    s = x.shape[0]
    tau = _bp64(torch.ones_like(b[:1]), n, degs).abs() + 4.0
    tau = 0.95 / torch.where(tau / tau.amax() < 1e-5, torch.ones_like(tau), tau)
    sig = _fp64(torch.ones_like(x), map_of, 1, degs).abs()
    sig = 0.95 / torch.where(sig / sig.amax(dim=(1, 2, 3), keepdim=True) < 1e-5, torch.ones_like(sig), sig)
    p, q, xr = torch.zeros_like(b), torch.zeros((s, 2, n, n), dtype=torch.float64, device=b.device), x
    for _ in range(case["iterations"]):
        p = p + _fp64(xr, map_of, 1, degs) * sig
        p = (1 + p - torch.sqrt((p - 1) ** 2 + 4 * sig * b)) / 2
        q[:, 0, :-1] += 0.5 * (xr[:, 1:] - xr[:, :-1])
        q[:, 1, :, :-1] += 0.5 * (xr[:, :, 1:] - xr[:, :, :-1])
        q = q / torch.clamp(torch.sqrt((q * q).sum(1, keepdim=True)), min=1e-2) * 1e-2
        div = torch.zeros_like(x)
        div[:, 1:] += q[:, 0, 1:] - q[:, 0, :-1]
        div[:, :, 1:] += q[:, 1, :, 1:] - q[:, 1, :, :-1]
        xn = torch.clamp(x - (_bp64(p, n, degs) - div) * tau, min=0.0)
        xr, x = 2 * xn - x, xn
    return x


def _conv64(x, w, bias=None):
    """x NCHW FP64, w (cout, 9, cin)."""
    w = w.double().reshape(w.shape[0], 3, 3, w.shape[2]).permute(0, 3, 1, 2).contiguous()
    return torch.nn.functional.conv2d(x, w, None if bias is None else bias.double(), padding=1)


def _net64(x):
    p = {k: tuple(v.to(x.device) for v in t) for k, t in torch.load(WEIGHTS, map_location="cpu").items()
         if isinstance(t, tuple)}

    def conv(name, v, relu=True):
        v = _conv64(v, *p[name])
        return v.relu() if relu else v

    def pool(v):
        return torch.nn.functional.avg_pool2d(v, 2)

    def up(v):
        return torch.nn.functional.interpolate(v, scale_factor=2, mode="nearest")

    outs = []
    for one in x:
        v = one[None].permute(0, 3, 1, 2).double()
        e1 = conv("e1b", conv("e1a", v))
        e2 = conv("e2b", conv("e2a", pool(e1)))
        e3 = conv("e3b", conv("e3a", pool(e2)))
        bt = conv("b2", conv("b1", pool(e3)))
        d3 = conv("d3b", conv("d3a", up(bt)) + e3)
        d2 = conv("d2b", conv("d2a", up(d3)) + e2)
        d1 = conv("d1b", conv("d1a", up(d2)) + e1)
        outs.append(conv("head", d1, False).permute(0, 2, 3, 1))
    return torch.cat(outs).contiguous()


def _conv_backward64(t):
    x, dy = (t[k].permute(0, 3, 1, 2).double() for k in ("x", "dy"))
    h, w = x.shape[2:]
    xp = torch.nn.functional.pad(x, (1, 1, 1, 1))
    rows = dy.permute(1, 0, 2, 3).reshape(dy.shape[1], -1)
    dw = torch.stack([rows @ xp[:, :, ky:ky + h, kx:kx + w].permute(0, 2, 3, 1).reshape(-1, x.shape[1])
                      for ky in range(3) for kx in range(3)], 1)
    wf = t["w"].double().flip(1).permute(2, 1, 0)
    return dw, rows.sum(1), _conv64(dy, wf).permute(0, 2, 3, 1).contiguous()


def exact(case, seed):
    kind, t = case["kind"], _inputs(case, seed)
    if kind in ("project", "adjoint"):
        n, d, degs = case["n"], case["dets"], _degrees(_angles(case["angles"]))
        map_of = lambda a: t["maps"][:, a].double()  # noqa: E731
        y = t["y"].double()[None]
        if kind == "adjoint":
            return _adjoint64(y, n, degs, map_of)
        fp = _fp64(t["x"].double()[None], map_of, d, degs)[0]
        return (fp if d > 1 else fp[0]), _bp64(y, n, degs)[0]
    if kind in ("mlem", "mlem_call"):
        degs = _degrees(_angles(case["angles"]))
        x, res = _mlem64(t["b"], case["n"], degs, lambda a: t["maps"][:, a].double(), case["iterations"])
        if kind == "mlem":
            return x, res[-1]
        return x[0], torch.stack(res)[:, 0]
    if kind == "subsets":
        degs, x, at = _degrees(t["angles"]), None, 0
        for r in range(case["subsets"]):
            k = len(range(r, case["angles"], case["subsets"]))
            x, _ = _mlem64(t["b"][:, :, at:at + k], case["n"], degs[at:at + k],
                           lambda a, at=at: t["maps"][:, at + a].double(), 1, x)
            at += k
        return x
    if kind == "maps":
        return _maps64(case, t)
    if kind == "pdhg":
        return _pdhg64(case, t)
    if kind == "ragged":
        outs = []
        for g in t["groups"]:
            degs = _degrees(_angles(g["angles"]))
            map_of = lambda a, m=g["maps"]: m[:, a].double()  # noqa: E731
            b, x, n = g["b"].double(), g["x0"].double(), g["n"]
            tau = _bp64(torch.ones_like(b), n, degs, map_of).abs()
            tau = 1 / torch.where(tau / tau.amax(dim=(1, 2), keepdim=True) < 1e-5, torch.ones_like(tau), tau)
            sig = _fp64(torch.ones_like(x), map_of, 1, degs).abs()
            sig = 1 / torch.where(sig / sig.amax(dim=(1, 2, 3), keepdim=True) < 1e-5, torch.ones_like(sig), sig)
            upd = _bp64((b - _fp64(x, map_of, 1, degs)) * sig, n, degs, map_of)
            outs.append(torch.clamp(x + upd * tau, min=0.0))
        return outs
    if kind == "net":
        return _net64(t["x"])
    return _conv_backward64(t)
