"""Performance cases: the work a user has the library do, through its public entry points.

Each case is one call of a kind below, on seeded synthetic list-mode data (a cylinder
phantom with hot spheres seen by a ring scanner; no dataset is involved):

* ``step``: projection of an image along TOF events and the back-projection of its values
  (``projection_backprojection``), what one MLEM update or one OSEM subset costs;
* ``project`` / ``backproject``: each direction by itself;
* ``gradient``: loss and image gradient of a Poisson likelihood (autograd: projection
  forward, plain adjoint backward);
* ``osem``: a reconstruction from preprocessed events (subsets, record order, one pass);
* ``batched``: one iteration of many frames at once, replayed as a CUDA graph;
* ``map`` / ``map_generated``: the efficiency map's sum over detector pairs, from a tensor
  of pairs or from pairs that the kernels make themselves;
* ``siddon``: the ray-tracing step, TOF off or on;
* ``preprocess``: raw events to the records of the three axis groups.

``exact`` restates every kind in float64 with plain torch operations.
"""

import math

import numpy as np
import torch

FWHM = 2.35482005
KW_4MM = 6 * 4.0 / FWHM  # a tube of 4 mm FWHM, six sigma wide
DEV = "cuda"
AXES = ("x", "y", "z")
# kernel axes of each dominant-axis group, fastest first (world axes 0, 1, 2)
KERNEL_AXES = {"x": (1, 2, 0), "y": (0, 2, 1), "z": (0, 1, 2)}
NO_TOF = 1.0e6  # ps: the variance is far above the value at which TOF switches off


def _case(name, kind, grid, voxel, events, tof=530.0, kw=KW_4MM, geo=False, ring=400, rings=32,
          pitch=3.2, radius=400.0, body=100.0, ordered=False, **more):
    return dict(name=name, kind=kind, nx=grid[0], ny=grid[1], nz=grid[2], voxel=voxel,
                events=events, tof=tof, kw=kw, geo=geo, ring=ring, rings=rings, pitch=pitch,
                radius=radius, body=body, ordered=ordered, **more)


def listed():
    return [
        # a preview or a short gate: so few events that latency and launches are what counts
        _case("step_tiny", "step", (64, 64, 32), 6.4, 2_000),
        # a short frame on a grid of no round size, with the preset tube width of 4 mm and
        # its geometric scaling, without TOF
        _case("project_odd", "project", (101, 93, 47), 3.7, 60_001, tof=NO_TOF, kw=4.0, geo=True),
        # one subset's size of events, back-projection alone
        _case("backproject_128", "backproject", (128, 128, 64), 3.2, 400_000),
        # the headline step: 10M events at 530 ps, records grouped by direction
        _case("step_128", "step", (128, 128, 64), 3.2, 10_000_000, ordered=True),
        # a long axial field of view: 1 m of rings, 400 ps, part of a streamed chunk
        _case("step_256", "step", (256, 256, 128), 2.5, 4_000_000, tof=400.0, ring=600, rings=320,
              pitch=3.125, radius=390.0, body=200.0, ordered=True),
        # gradient-based reconstruction: one frame's likelihood and its gradient
        _case("gradient_128", "gradient", (128, 128, 64), 3.2, 1_000_000),
        # a whole reconstruction pass from preprocessed events
        _case("osem_128", "osem", (128, 128, 64), 3.2, 1_000_000, subsets=10),
        # dynamic frames with uneven event counts, advanced together
        _case("batched_96", "batched", (96, 96, 48), 3.2, 4_000_000, frames=16, subsets=5),
        # the sensitivity pass over random detector pairs
        _case("map_128", "map", (128, 128, 64), 3.2, 6_000_000),
        # the same for the long scanner, pairs made on the device
        _case("map_generated_256", "map_generated", (256, 256, 128), 2.5, 3_000_000, ring=600,
              rings=320, pitch=3.125, radius=390.0),
        # ray tracing without TOF: the plain list-mode step
        _case("siddon_64", "siddon", (64, 64, 32), 3.4, 1_000_000, tof=NO_TOF),
        # raw events to preprocessed records
        _case("preprocess", "preprocess", (128, 128, 64), 3.2, 8_000_000),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("step", "step", "project", "backproject", "gradient", "osem", "batched",
                       "map", "map_generated", "siddon", "siddon", "preprocess"))
    most = {"step": 4e6, "project": 4e6, "backproject": 4e6, "gradient": 1e6, "osem": 1e6,
            "batched": 2e6, "map": 4e6, "map_generated": 2e6, "siddon": 2e6, "preprocess": 8e6}
    voxel = rng.choice((2.5, 3.0, 3.2, 3.4, 3.7, 4.0, 5.1, 6.4))
    # square fields of view of 190 to 640 mm, at most 256 voxels wide
    most_wide = 450.0 if kind in ("osem", "batched") else 640.0
    wide = rng.uniform(190.0, min(most_wide, 256 * voxel))
    nx = max(32, int(round(wide / voxel)))
    ny = max(32, nx - rng.choice((0, 0, 0, 1, 3, 8)))
    long_axis = rng.random() < 0.25 and kind not in ("osem", "batched")
    scanner = (dict(ring=600, rings=320, pitch=3.125, radius=390.0) if long_axis else
               dict(ring=400, rings=32, pitch=3.2, radius=400.0))
    axial = scanner["rings"] * scanner["pitch"]
    # long scanner: up to 128 slices; short: about its length or twice that
    nz = log_int(48, 128) if long_axis else max(16, int(round(axial * rng.choice((1, 2)) / voxel)))
    c = _case(None, kind, (nx, ny, nz), voxel, log_int(2e3 if kind != "preprocess" else 2e4, most[kind]),
              tof=rng.choice((400.0, 530.0, 530.0, NO_TOF)) if kind not in ("batched", "osem")
              else rng.choice((400.0, 530.0)),
              kw=rng.choice((KW_4MM, KW_4MM, 4.0, 8.0)), geo=rng.random() < 0.25,
              body=rng.uniform(0.3, 0.45) * wide, ordered=rng.random() < 0.5, **scanner)
    if c["tof"] == NO_TOF:  # uncut LORs cross the whole field of view
        c["events"] = min(c["events"], 1_000_000)
    if kind in ("osem", "batched"):
        # enough events in every subset that each updates most of the object's voxels
        c["subsets"] = rng.choice((1, 4, 7, 10) if kind == "osem" else (2, 5))
        if kind == "batched":
            c["frames"] = rng.randint(2, 12)
        c["events"] = max(c["events"], 40_000 * c["subsets"] * c.get("frames", 1))
    del c["name"]
    return c


# ------------------------------------------------------------------------------- inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _size(c):
    return [c["nx"] * c["voxel"], c["ny"] * c["voxel"], c["nz"] * c["voxel"]]


def _grid(c):
    return [c["nx"], c["ny"], c["nz"]]


def _tof(c):
    """(tof_bin, tof_sigma2) in mm, mm^2: a 40 ps bin and the resolution's sigma."""
    return 6.0, (c["tof"] * 0.15 / FWHM) ** 2


def _crystal(c, k, j):
    phi = k.double() * (2 * math.pi / c["ring"])
    z = (j.double() - (c["rings"] - 1) / 2) * c["pitch"]
    return torch.stack([c["radius"] * torch.cos(phi), c["radius"] * torch.sin(phi), z],
                       -1).float()


def _axis_of(ev):
    """The dominant axis of each event (0, 1, 2), by float32 differences."""
    d = (ev[:, 3:6] - ev[:, 0:3]).abs()
    x = (d[:, 0] >= d[:, 1]) & (d[:, 0] >= d[:, 2])
    return torch.where(x, 0, torch.where((d[:, 1] > d[:, 0]) & (d[:, 1] >= d[:, 2]), 1, 2))


def _events(c, n, g):
    """[n, 7] float32 events (two crystal centres, TOF position) of the phantom, with the
    same number in each axis group for every seed: half x, half y, on the long scanner 2 %
    (about what it sees) along z."""
    along = n // 50 if c["rings"] > 100 else 0
    quota = [(n - along + 1) // 2, (n - along) // 2, along]
    parts, left = [], list(quota)
    while sum(left):
        ev = _some_events(c, max(1024, int(1.05 * max(2 * left[0], 2 * left[1], 60 * left[2]))), g)
        axis = _axis_of(ev)
        keep = torch.zeros(len(ev), dtype=torch.bool, device=DEV)
        for k in range(3):
            at = torch.nonzero(axis == k)[: left[k], 0]
            keep[at] = True
            left[k] -= len(at)
        parts.append(ev[keep])
    return torch.cat(parts).contiguous()


def _some_events(c, n, g):
    R, r = c["radius"], min(c["body"], 0.9 * c["radius"])
    axial = c["rings"] * c["pitch"]
    half = min(axial, _size(c)[2]) / 2
    slope = axial / (2 * math.sqrt(R * R - r * r))  # no steeper line has both ends on the rings
    cmax = slope / math.sqrt(1 + slope * slope)
    out, have = [], 0
    while have < n:
        m = min(1 << 22, int((n - have) * 2.2) + 1024)
        u = torch.rand(6, m, generator=g, device=DEV, dtype=torch.float64)
        rho, ang = r * torch.sqrt(u[0]), 2 * math.pi * u[1]
        # one event in ten from four hot balls of 0.08 r, the rest from the cylinder
        hot = u[5] < 0.1
        ball = torch.floor(u[0] * 4) * (math.pi / 2)
        rho_h = 0.08 * r * torch.rand(m, generator=g, device=DEV, dtype=torch.float64) ** (1 / 3)
        x = torch.where(hot, 0.5 * r * torch.cos(ball) + rho_h * torch.cos(ang), rho * torch.cos(ang))
        y = torch.where(hot, 0.5 * r * torch.sin(ball) + rho_h * torch.sin(ang), rho * torch.sin(ang))
        z = (2 * u[2] - 1) * torch.where(hot, 0.25 * half, half)
        ct = (2 * u[3] - 1) * cmax
        st, az = torch.sqrt(1 - ct * ct), 2 * math.pi * u[4]
        dx, dy = st * torch.cos(az), st * torch.sin(az)
        a, b = st * st, x * dx + y * dy
        root = torch.sqrt(b * b - a * (x * x + y * y - R * R))
        ends, ok = [], None
        for t in ((-b - root) / a, (-b + root) / a):
            k = torch.round(torch.atan2(y + t * dy, x + t * dx) * (c["ring"] / (2 * math.pi)))
            j = torch.round((z + t * ct) / c["pitch"] + (c["rings"] - 1) / 2)
            inside = (j >= 0) & (j < c["rings"])
            ok = inside if ok is None else ok & inside
            ends.append((k.remainder(c["ring"]), j))
        p = torch.stack([x, y, z], 1)[ok]
        e1, e2 = (_crystal(c, k[ok], j[ok]) for k, j in ends)
        d = (e2 - e1).double()
        L = d.norm(dim=1)
        t = L / 2 - ((p - e1.double()) * d).sum(1) / L
        sigma = math.sqrt(_tof(c)[1]) if c["tof"] < NO_TOF else 0.0
        t = t + sigma * torch.randn(t.shape[0], generator=g, device=DEV, dtype=torch.float64)
        out.append(torch.cat([e1, e2, t.float()[:, None]], 1))
        have += out[-1].shape[0]
    return torch.cat(out)[:n].contiguous()


def _split(ev, recon, limit, dtype):
    """The preprocessing of events in plain torch: {'x','y','z'} records (dominant axis last,
    endpoints in its ascending direction, TOF centre and cut), values in ``dtype``."""
    d32, ax = ev[:, 3:6] - ev[:, 0:3], _axis_of(ev)
    swap = ~(d32.gather(1, ax[:, None])[:, 0] >= 0)
    e = ev.to(dtype)
    p1, p2 = e[:, 0:3], e[:, 3:6]
    d = p2 - p1
    dsq = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
    rsq = (p1[:, 0] * p1[:, 0] + p2[:, 0] * p2[:, 0]) + p1[:, 1] * p1[:, 1] + p2[:, 1] * p2[:, 1]
    f = dsq * dsq / rsq / (dsq + d[:, 2] * d[:, 2]) / 2
    s = swap[:, None]
    p1, p2 = torch.where(s, p2, p1), torch.where(s, p1, p2)
    cols = [p1, p2]
    if recon:
        t = torch.where(swap, 0 - e[:, 6], e[:, 6])
        pd = p2 - p1
        L = torch.sqrt(pd[:, 0] * pd[:, 0] + pd[:, 1] * pd[:, 1] + pd[:, 2] * pd[:, 2])
        u = pd / L[:, None]
        mid = (0.5 - t / L)[:, None] * pd + p1
        off = mid - p1
        far = torch.sqrt(off[:, 0] * off[:, 0] + off[:, 1] * off[:, 1] + off[:, 2] * off[:, 2])
        cut = (far > limit)[:, None] if limit is not None else torch.zeros_like(s)
        lim = 0.0 if limit is None else limit
        cols = [torch.where(cut, mid - lim * u, p1), torch.where(cut, mid + lim * u, p2), mid]
    rank = ax * 2 + swap.long()
    groups = {}
    for k, a in enumerate(AXES):
        at = torch.cat([torch.nonzero(rank == 2 * k)[:, 0], torch.nonzero(rank == 2 * k + 1)[:, 0]])
        groups[a] = torch.cat([v[at][:, list(KERNEL_AXES[a])] for v in cols]
                              + [f[at][:, None]], 1).contiguous()
    return groups


def _limit(c, dtype):
    if c["tof"] >= 1.0e4:
        return None
    lim = c["tof"] * 0.15 / FWHM * 3
    return float(np.float32(lim)) if dtype == torch.float32 else lim


def _by_direction(rec):
    """Records grouped by direction inside runs of 4096, as a reconstruction orders them."""
    d = rec[:, 3:6] - rec[:, 0:3]
    u2 = (d / d.norm(dim=1, keepdim=True)) ** 2
    q = (1 - u2[:, 0] - u2[:, 1]).clamp(min=1e-6)
    kx = ((((1 - u2[:, 1]) / q).sqrt() - 1) * 16).long().clamp(0, 15)
    ky = ((((1 - u2[:, 0]) / q).sqrt() - 1) * 16).long().clamp(0, 15)
    kz = ((torch.minimum(rec[:, 2], rec[:, 5]) + 1024) * 0.125).long().clamp(0, 255)
    run = torch.arange(rec.shape[0], device=rec.device) // 4096
    return rec[torch.argsort(run * (1 << 17) + (kx * 16 + ky) * 256 + kz, stable=True)].contiguous()


def _records(c, n, g):
    """Preprocessed TOR records of n events, grouped by direction where the case says so."""
    groups = _split(_events(c, n, g), True, _limit(c, torch.float32), torch.float32)
    return {a: _by_direction(r) if c["ordered"] and len(r) > 1 else r for a, r in groups.items()}


def _mesh(c):
    s, n = _size(c), _grid(c)
    ax = [(torch.arange(n[k], device=DEV, dtype=torch.float32) + 0.5) * c["voxel"] - s[k] / 2
          for k in range(3)]
    return torch.meshgrid(*ax, indexing="ij")


def _image(c, g):
    """An iterate of a reconstruction: the phantom with noise over a faint background."""
    x, y, _ = _mesh(c)
    r = min(c["body"], 0.9 * c["radius"])
    img = 0.02 + (x * x + y * y <= r * r).float()
    for k in range(4):
        hx, hy = 0.5 * r * math.cos(k * math.pi / 2), 0.5 * r * math.sin(k * math.pi / 2)
        img += 3.0 * ((x - hx) ** 2 + (y - hy) ** 2 <= (0.08 * r + c["voxel"]) ** 2)
    return (img * (1 + 0.1 * torch.rand(img.shape, generator=g, device=DEV))).contiguous()


def _effinv(c):
    """A smooth inverted efficiency map and the matching initial image (ones in its support)."""
    x, y, z = _mesh(c)
    keep = (x * x + y * y <= (0.49 * c["nx"] * c["voxel"]) ** 2).float()
    return keep / (1.0 - 0.8 * z.abs() / z.abs().max()) / 50.0, keep.contiguous()


def _frames(c, g):
    """Event counts of the frames: log-uniform over a factor of 25, scaled to the total."""
    w = torch.exp(torch.rand(c["frames"], generator=g, device=DEV) * math.log(25.0)).cpu().double()
    return [max(50, int(v)) for v in w / w.sum() * c["events"]]


def _pairs(c, n, g):
    m = c["ring"] * c["rings"]
    i = torch.randint(0, m, (n,), generator=g, device=DEV)
    j = torch.randint(0, m - 1, (n,), generator=g, device=DEV)
    j = j + (j >= i)
    return torch.cat([_crystal(c, k % c["ring"], k // c["ring"]) for k in (i, j)], 1).contiguous()


# ------------------------------------------------------------------------------ the calls


def prepare(case, seed):
    from srf_b200 import CompleteLoRsModel, Image, ListModeData, SplitLoRsModel
    from srf_b200.preprocess import split_listmode

    c, g, kind = case, _gen(seed), case["kind"]
    bin_mm, s2 = _tof(c)
    center, size = [0.0, 0.0, 0.0], _size(c)
    if kind == "preprocess":
        return dict(kind=kind, events=_events(c, c["events"], g), tof=c["tof"])
    if kind == "siddon":
        model = CompleteLoRsModel(tof_sigma2=s2, tof_bin=bin_mm)
        ev = _events(c, c["events"], g)
        return dict(kind="step", model=model, image=Image(_image(c, g), center, size),
                    data=ListModeData(ev, torch.ones(len(ev), device=DEV)))
    model = SplitLoRsModel(c["kw"], c["geo"], tof_sigma2=s2, tof_bin=bin_mm)
    state = dict(kind=kind, model=model, grid=_grid(c), center=center, size=size)
    if kind == "map":
        return dict(state, lors=_pairs(c, c["events"], g))
    if kind == "map_generated":
        from srf_b200.scanner import RingScanner
        from srf_b200.synthetic import GeneratedPairs
        scanner = RingScanner(c["radius"], c["ring"], c["rings"], c["pitch"])
        return dict(state, kind="map", lors=GeneratedPairs.random(scanner, c["events"], seed))
    if kind == "batched":
        from srf_b200.batched import BatchedOSEM
        eff, x0 = _effinv(c)
        frames = [_records(c, n, g) for n in _frames(c, g)]
        osem = BatchedOSEM(model, frames, Image(eff, center, size), x0, c["subsets"],
                           use_graph=True)
        return dict(state, osem=osem, x0=x0)
    data = split_listmode(_records(c, c["events"], g))
    if kind == "osem":
        eff, x0 = _effinv(c)
        return dict(state, data=data, effinv=Image(eff, center, size),
                    x0=Image(x0, center, size), subsets=c["subsets"])
    image = Image(_image(c, g), center, size)
    if kind == "backproject":  # values of the range that a projection gives
        vals = {a: 1.0 + 40.0 * torch.rand(len(data[a]), generator=g, device=DEV) for a in AXES}
        data = split_listmode({a: data[a].lors for a in AXES}, vals)
    if kind == "gradient":
        from srf_b200.autograd import Projector
        return dict(state, projector=Projector(model, data, _grid(c), center, size),
                    x=image.data, sens=_sens(c, g))
    return dict(state, image=image, data=data)


def _sens(c, g):
    return 1.0 + torch.rand(_grid(c), generator=g, device=DEV)


def run(state):
    from srf_b200 import backprojection, projection, projection_backprojection, recon_process

    kind = state["kind"]
    if kind == "step":
        proj, back = projection_backprojection(state["model"], state["image"], state["data"])
        vals = [proj[a].values for a in AXES] if hasattr(proj, "x") else proj.values
        return {"values": vals, "back": back.data}
    if kind == "project":
        proj = projection(state["model"], state["image"], state["data"])
        return {"values": [proj[a].values for a in AXES]}
    if kind == "backproject":
        return {"back": backprojection(state["model"], state["data"], state["image"]).data}
    if kind == "preprocess":
        groups = recon_process(state["events"], state["tof"])
        return [groups[a] for a in AXES]
    if kind == "map":
        from srf_b200.recon import map_sum
        return map_sum(state["model"], state["lors"], state["grid"], state["center"],
                       state["size"])
    if kind == "osem":
        from srf_b200.recon import OSEM
        return OSEM(state["model"], state["data"], state["effinv"], state["x0"],
                    state["subsets"]).run(1).data
    if kind == "batched":
        osem = state["osem"]
        osem.x.copy_(state["x0"].expand_as(osem.x))  # from the initial image
        return osem.step()
    from srf_b200.autograd import poisson_nll, quadratic_penalty
    x = state["x"].detach().requires_grad_(True)
    p = state["projector"].forward(x)
    loss = poisson_nll(p, x, state["sens"]) + quadratic_penalty(x, 0.01)
    loss.backward()
    return {"loss": loss.detach(), "grad": x.grad}


# --------------------------------------------------------------------------------- work


def work(case):
    c, kind = case, case["kind"]
    n, vox = c["events"], c["nx"] * c["ny"] * c["nz"]
    if kind == "preprocess":
        return {"bytes": n * (28 + 40), "flops": n * 40}
    v, w = c["voxel"], min(c["nx"], c["ny"]) * c["voxel"]
    if kind == "siddon":  # voxels on a ray, 8 operations each, both directions
        seen = 1.5 * 0.8 * w / v
        return {"bytes": n * (2 * 28 + 8) + vox * 8, "flops": n * seen * 16}
    # voxels inside the tube: its section over the length inside the field of view
    length = 0.8 * w if c["tof"] >= 1.0e4 or kind.startswith("map") else min(
        0.8 * w, 6 * math.sqrt(_tof(c)[1]))
    samples = max(1.0, 0.85 * length / v * 1.2 * math.pi * (c["kw"] / 2 / v) ** 2)
    both = {"step": 2, "gradient": 2, "osem": 2, "batched": 2}.get(kind, 1)
    rec = 24 if kind == "map" else 0 if kind == "map_generated" else 40
    images = vox * 4 * (2 if both == 2 else 1) * c.get("frames", 1) * c.get("subsets", 1)
    return {"bytes": n * (rec + (4 if rec == 40 else 0)) + images,
            "flops": n * samples * 12 * both}


# ------------------------------------------------------------------ the same in float64


def _tor_items(c, rec, axis, tof, chunk=400_000):
    """The (LOR, slice) crossings of records in float64, a chunk of LORs at a time: yields
    (LOR index, voxels and weights one window position at a time)."""
    ka = KERNEL_AXES[axis]
    n = [_grid(c)[k] for k in ka]
    inter = [_size(c)[k] / _grid(c)[k] for k in ka]
    lo = [-_size(c)[k] / 2 for k in ka]
    patch = math.ceil((math.sqrt(2.0) * c["kw"] + inter[2]) / inter[0])
    stride = [_stride(c)[k] for k in ka]
    bin_mm, s2 = _tof(c)
    tof = tof and s2 < 405758.0
    planes = lo[2] + (torch.arange(n[2], device=DEV, dtype=torch.float64) + 0.5) * inter[2]
    for at in range(0, len(rec), chunk):
        r = rec[at:at + chunk].double()
        p, d = r[:, 0:3], r[:, 3:6] - r[:, 0:3]
        ratio = (planes[None, :] - p[:, 2:3]) / d[:, 2:3]
        lor, s = torch.nonzero((ratio > 0) & (ratio < 1), as_tuple=True)
        t = ratio[lor, s]
        del ratio
        u = d / d.norm(dim=1, keepdim=True)
        cx, cy = p[lor, 0] + t * d[lor, 0], p[lor, 1] + t * d[lor, 1]
        ux, uy = u[lor, 0], u[lor, 1]
        sig = c["kw"] ** 2 / 36 * (r[lor, -1] if c["geo"] else torch.ones_like(t))
        ix0 = torch.trunc((cx - lo[0]) / inter[0]).long() - patch // 2
        iy0 = torch.trunc((cy - lo[1]) / inter[1]).long() - patch // 2
        tse = s2 + bin_mm ** 2 / 12
        if tof:
            far = (r[lor, 6] - cx) ** 2 + (r[lor, 7] - cy) ** 2 + (r[lor, 8] - planes[s]) ** 2
        base = s * stride[2]
        for j in range(patch):
            iy = iy0 + j
            dy = cy - (lo[1] + (iy + 0.5) * inter[1])
            for i in range(patch):
                ix = ix0 + i
                dx = cx - (lo[0] + (ix + 0.5) * inter[0])
                d2 = dx * dx + dy * dy - (dx * ux + dy * uy) ** 2
                use = (d2 < 9 * sig) & (ix >= 0) & (ix < n[0]) & (iy >= 0) & (iy < n[1])
                e = -d2 / (2 * sig)
                if tof:
                    e = e - (far - d2) / (2 * tse)
                w = torch.where(use, torch.exp(e), torch.zeros_like(e))
                if tof:
                    w = w * (bin_mm / math.sqrt(2 * math.pi * s2))
                voxel = torch.where(use, base + iy * stride[1] + ix * stride[0],
                                    torch.zeros_like(base))
                yield at + lor, voxel, w


def _stride(c):
    return [c["ny"] * c["nz"], c["nz"], 1]


def _tor_project(c, groups, img):
    flat, out = img.double().reshape(-1), {}
    for a in AXES:
        v = torch.zeros(len(groups[a]), device=DEV, dtype=torch.float64)
        for lor, voxel, w in _tor_items(c, groups[a], a, True):
            v.index_add_(0, lor, w * flat[voxel])
        out[a] = v
    return out


def _tor_back(c, groups, scale, tof=True):
    """Sum of w * scale over the groups' LORs, [nx, ny, nz] float64."""
    img = torch.zeros(c["nx"] * c["ny"] * c["nz"], device=DEV, dtype=torch.float64)
    for a in AXES:
        for lor, voxel, w in _tor_items(c, groups[a], a, tof):
            img.index_add_(0, voxel, w * scale[a][lor])
    return img.reshape(_grid(c))


def _inverse(v):
    return {a: torch.where(x > 1e-7, 1.0 / x.clamp(min=1e-30), torch.zeros_like(x))
            for a, x in v.items()}


def _em(c, groups, eff, x, subsets):
    for k in range(subsets):
        part = {a: groups[a][k::subsets] for a in AXES}
        x = x * (eff * subsets) * _tor_back(c, part, _inverse(_tor_project(c, part, x)))
    return x


def _siddon(c, ev, img, chunk=100_000):
    """(projected values, back-projection of them) of a ray step, by sorted plane crossings."""
    n, h = _grid(c), [s / 2 for s in _size(c)]
    bin_mm, s2 = _tof(c)
    flat = img.double().reshape(-1)
    back, values = torch.zeros_like(flat), []
    for at in range(0, len(ev), chunk):
        e = ev[at:at + chunk].double()
        p, d = e[:, 0:3], e[:, 3:6] - e[:, 0:3]
        L = d.norm(dim=1)
        u = d / L[:, None]
        t0, t1, cuts = torch.zeros_like(L), L, []
        for k in range(3):
            pl = torch.linspace(-h[k], h[k], n[k] + 1, device=DEV, dtype=torch.float64)
            par = u[:, k] == 0
            t = (pl[None, :] - p[:, k:k + 1]) / torch.where(par, torch.ones_like(L), u[:, k])[:, None]
            first, last = torch.minimum(t[:, 0], t[:, -1]), torch.maximum(t[:, 0], t[:, -1])
            out = par & (p[:, k].abs() > h[k])
            t0 = torch.where(par, t0, torch.maximum(t0, first))
            t1 = torch.where(out, torch.zeros_like(t1), torch.where(par, t1, torch.minimum(t1, last)))
            cuts.append(torch.where(par[:, None], torch.zeros_like(t), t))
        t = torch.cat(cuts, 1)
        t1 = torch.maximum(t0, t1)
        t = torch.sort(torch.minimum(torch.maximum(t, t0[:, None]), t1[:, None]), 1)[0]
        length, mid = t[:, 1:] - t[:, :-1], (t[:, 1:] + t[:, :-1]) / 2
        voxel = torch.zeros_like(mid, dtype=torch.int64)
        for k in range(3):
            i = torch.floor((p[:, k:k + 1] + mid * u[:, k:k + 1] + h[k]) / c["voxel"]).long()
            voxel += i.clamp(0, n[k] - 1) * _stride(c)[k]
        w = length / (L * L)[:, None]
        if s2 < 405758.0:
            tt = (L / 2 - e[:, 6])[:, None] - mid
            var = s2 + (length * length + bin_mm ** 2) / 12
            r = tt * tt / var
            w = torch.where(r < 9, w * bin_mm * torch.exp(-r / 2) / torch.sqrt(2 * math.pi * var),
                            torch.zeros_like(w))
        v = (w * flat[voxel]).sum(1)
        back.index_add_(0, voxel.reshape(-1),
                        (w * torch.where(v > 0, 1 / v, torch.zeros_like(v))[:, None]).reshape(-1))
        values.append(v)
    return torch.cat(values), back.reshape(n)


def _chords(c, count, seed):
    """The random chords of a generated map (SplitMix64 draws by LOR number), [count, 6]."""
    def mix(k):
        z = np.uint64(seed) + (k + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    def part(u, m):
        return ((u * m) >> np.uint64(32)).astype(np.int64)

    n, nr, low = c["ring"], c["rings"], np.uint64(0xFFFFFFFF)
    with np.errstate(over="ignore"):
        g = np.arange(count, dtype=np.uint64)
        group, i = g // np.uint64(256), g % np.uint64(256)
        h1, h2 = mix(np.uint64(4) * group), mix(np.uint64(4) * group + np.uint64(2))
        s = part(h1 >> np.uint64(32), np.uint64(n))
        d = part(h2 >> np.uint64(32), np.uint64(nr)) - part(h1 & low, np.uint64(nr))
        h = mix(np.uint64(2) * g + np.uint64(1))
        a = ((((i << np.uint64(32)) | (h >> np.uint64(32))) * np.uint64(n)) >> np.uint64(40))
        a = a.astype(np.int64)
        ra = np.maximum(0, -d) + part(h & low, (nr - np.abs(d)).astype(np.uint64))
    b, rb = (s + n - a) % n, ra + d
    keep = (a != b) | (ra != rb)
    to = [torch.as_tensor(v[keep], device=DEV) for v in (a, ra, b, rb)]
    return torch.cat([_crystal(c, to[0], to[1]), _crystal(c, to[2], to[3])], 1)


def exact(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    if kind == "preprocess":
        groups = _split(_events(c, c["events"], g), True, _limit(c, torch.float64), torch.float64)
        return [groups[a] for a in AXES]
    if kind == "siddon":
        ev = _events(c, c["events"], g)
        values, back = _siddon(c, ev, _image(c, g))
        return {"values": values, "back": back}
    if kind in ("map", "map_generated"):
        lors = _pairs(c, c["events"], g) if kind == "map" else _chords(c, c["events"], seed)
        groups = _split(lors, False, None, torch.float32)
        ones = {a: torch.ones(len(groups[a]), device=DEV, dtype=torch.float64) for a in AXES}
        return _tor_back(c, groups, ones, tof=False)
    if kind == "batched":
        eff, x0 = (v.double() for v in _effinv(c))
        frames = [_records(c, n, g) for n in _frames(c, g)]
        return torch.stack([_em(c, f, eff, x0, c["subsets"]) for f in frames])
    groups = _records(c, c["events"], g)
    if kind == "osem":
        eff, x0 = (v.double() for v in _effinv(c))
        return _em(c, groups, eff, x0, c["subsets"])
    img = _image(c, g)
    if kind == "backproject":
        vals = {a: 1.0 + 40.0 * torch.rand(len(groups[a]), generator=g, device=DEV) for a in AXES}
        return {"back": _tor_back(c, groups, _inverse({a: v.double() for a, v in vals.items()}))}
    v = _tor_project(c, groups, img)
    if kind == "project":
        return {"values": [v[a] for a in AXES]}
    if kind == "step":
        return {"values": [v[a] for a in AXES], "back": _tor_back(c, groups, _inverse(v))}
    x, sens = img.double(), _sens(c, g).double()
    logs = sum(torch.log(p.clamp(min=1e-30)).sum() for p in v.values())
    inv = {a: torch.where(p > 1e-30, 1 / p.clamp(min=1e-30), torch.zeros_like(p))
           for a, p in v.items()}
    grad = sens - _tor_back(c, groups, inv)
    loss = (sens * x).sum() - logs
    for k in range(3):
        d = x.narrow(k, 1, x.shape[k] - 1) - x.narrow(k, 0, x.shape[k] - 1)
        loss = loss + 0.005 * (d * d).sum()
        grad.narrow(k, 1, x.shape[k] - 1).add_(0.01 * d)
        grad.narrow(k, 0, x.shape[k] - 1).sub_(0.01 * d)
    return {"loss": loss.float(), "grad": grad}
