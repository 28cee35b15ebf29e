"""Performance cases: the solver's public entry points over the sizes they are used at.

Each case is a plain dict.  ``kind`` names the entry point:

  solve       one ``steady_state_transport_solver`` call, numpy in and out
  batch       ``BatchSolver.solve``: many footprints, outputs left on the device
  batch_host  ``solve_batch``: the same with numpy outputs
  timeseries  ``vertical_profiles_batch`` and ``solve_stream`` over a met series, numpy out
  surrogate   ``Surrogate.solve_batch_prepared``: footprints through the trained network
  train       ``MLP.train_step``: one Adam step on the tensor cores
  points      ``point_measurement_batch``: footprint-weighted sums of flux fields

Sizes follow the repository's fixtures (64 x 128 and 64 x 32 grids, 16 levels), its
benchmark (512 x 512 footprint, 128 levels below z_m), its production configuration
(512 x 512 with a 500 m halo, all 1024 x 1024 modes, 256 levels) and its towers
(256, 512 and 1024 grids).  Met inputs are drawn from the seed.
"""

import functools
import math

import numpy as np
import torch

KAPPA = 0.4
DEV = "cuda" if torch.cuda.is_available() else "cpu"
# (grid, levels below z_m, domain in m) of the mixed batch's towers
TOWERS = [(256, 64, 1000.0), (512, 128, 1000.0), (1024, 256, 2000.0), (256, 96, 600.0), (512, 160, 1500.0),
          (256, 200, 800.0), (1024, 128, 3000.0), (512, 256, 1200.0)]


def _solve(name, mode, nx, ny, dx, n, zm, modes, halo, footprint, nlev, precision, shift):
    return dict(name=name, kind="solve", mode=mode, nx=nx, ny=ny, dx=dx, n=n, zm=zm, mx=modes[0], my=modes[1],
                halo=halo, footprint=footprint, nlev=nlev, precision=precision, shift=shift)


def listed():
    return [
        # the reference's own fixture size through the default mode: one tower, one time, latency
        _solve("footprint_fixture", "fp64", 64, 128, 5.0, 16, 10.0, (64, 128), -1.0, True, 1, "single", True),
        # the benchmark's footprint through the default mode (the reference's rounding)
        _solve("footprint_512", "fp64", 512, 512, 1000.0 / 512, 128, 20.0, (512, 512), -1.0, True, 1, "double", True),
        # a dispersion plume at nine heights, default mode, a grid that is no power of two
        _solve("plume_levels", "fp64", 190, 150, 4.0, 32, 10.0, (190, 150), -1.0, False, 9, "double", True),
        # the production footprint in the accurate FP64 mode (tall tower, fine grid, every mode)
        _solve("footprint_accurate", "fp64r", 512, 512, 1000.0 / 512, 256, 20.0, (1024, 1024), 500.0, True, 1,
               "single", True),
        # an interactive FP32 footprint, one call at a time
        _solve("footprint_fp32", "fp32", 256, 256, 1000.0 / 256, 64, 20.0, (256, 256), -1.0, True, 1, "single", True),
        # a day of half-hourly footprints of one tower: profiles, then batches of 16 in flight
        dict(name="timeseries_48", kind="timeseries", steps=48, nx=96, ny=128, dx=4.0, n=24, zm=12.0, mx=96, my=128),
        # the benchmark's step: 16 footprints of one tower, outputs left on the device
        dict(name="batch_512", kind="batch", count=16, nx=512, ny=512, dx=1000.0 / 512, n=128, zm=20.0, mx=512, my=512,
             nlev=1, footprint=True),
        # a batch over towers of different grids and level counts, results on the host
        dict(name="batch_towers", kind="batch_host", count=16, nx=0, ny=0, dx=0.0, n=0, zm=0.0, mx=0, my=0, nlev=1,
             footprint=True),
        # plumes of several sources at nine heights in FP32, outputs left on the device
        dict(name="batch_plumes", kind="batch", count=4, nx=256, ny=192, dx=4.0, n=64, zm=16.0, mx=256, my=192, nlev=9,
             footprint=False),
        # the benchmark's footprints through the trained network
        dict(name="surrogate_512", kind="surrogate", count=16, nx=512, ny=512, dx=1000.0 / 512),
        # one training step of the network at its training batch
        dict(name="train_65536", kind="train", samples=65536),
        # a footprint climatology against flux maps: 64 fields of 512 x 512
        dict(name="points_64", kind="points", count=64, nx=512, ny=512),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(v):
    return max(2, v - v % 2)


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "batch_host", "timeseries", "surrogate", "train", "points"])
    if kind == "train":
        return dict(kind=kind, samples=256 * _logint(rng, 4, 256))
    if kind == "points":
        return dict(kind=kind, count=_logint(rng, 1, 64), nx=_logint(rng, 64, 512), ny=_logint(rng, 64, 512))
    if kind == "surrogate":
        nx, ny = _logint(rng, 128, 512), _logint(rng, 128, 512)
        return dict(kind=kind, count=rng.randint(1, 16), nx=nx, ny=ny, dx=rng.uniform(2.0, 4.0))
    nx, ny, n = _logint(rng, 48, 512), _logint(rng, 48, 512), _logint(rng, 16, 128)
    footprint = rng.random() < 0.6
    dx = rng.uniform(2.0, 6.0)
    halo = -1.0 if rng.random() < 0.7 else round(rng.uniform(0.3, 1.0) * dx * max(nx, ny), 1)
    if not footprint:  # a source's truncated spectrum needs an even grid
        nx, ny = _even(nx), _even(ny)
    mx, my = _even(nx), _even(ny)
    zm = round(rng.uniform(3.0, 5.0) * dx, 2)
    if kind == "timeseries":
        return dict(kind=kind, steps=rng.randint(4, 48), nx=min(nx, 192), ny=min(ny, 192), dx=dx, n=min(n, 64), zm=zm,
                    mx=_even(min(nx, 192)), my=_even(min(ny, 192)))
    if kind in ("batch", "batch_host"):
        big = nx * ny > 256 * 256
        count = rng.randint(1, 8 if big else 16)
        return dict(kind=kind, count=count if footprint else min(count, 4), nx=nx, ny=ny, dx=dx, n=n, zm=zm, mx=mx,
                    my=my, nlev=1 if footprint else rng.choice([1, 5, 9]), footprint=footprint)
    mode = rng.choice(["fp64", "fp64", "fp64r", "fp32"])
    c = _solve("", mode, nx, ny, dx, n, zm, (mx, my), halo, footprint, 1 if footprint else rng.choice([1, 3, 9]),
               rng.choice(["single", "double"]), footprint or rng.random() < 0.7)
    del c["name"]
    return c


# --------------------------------------------------------------------------- inputs


def _psi(x):
    if x > 0:
        return 5.0 * x
    xi = (1.0 - 16.0 * x) ** 0.25
    return -2.0 * math.log(0.5 * (1 + xi)) - math.log(0.5 * (1 + xi * xi)) + 2.0 * math.atan(xi) - 0.5 * math.pi


def _profiles(n, zm, wind, ustar, mol):
    """MOST profiles on the log-stretched grid (default stretch and top)."""
    um, vm = wind
    absum = math.hypot(um, vm)
    z0 = zm * math.exp(-KAPPA * absum / ustar + _psi(zm / mol))
    h = 2.0 * zm
    bb = zm / (math.exp(-z0 / h) - math.exp(-zm / h))
    aa = bb * math.exp(-z0 / h)
    dzeta = zm / n
    zeta = np.arange(0.0, aa - bb * math.exp(-2.0 * zm / h) + dzeta, dzeta)
    z = -h * np.log(-(zeta - aa) / bb)
    x = z / mol
    if mol > 0:
        psi, phi = 5.0 * x, 1.0 + 5.0 * x
    else:
        xi = (1.0 - 16.0 * x) ** 0.25
        psi = -2.0 * np.log(0.5 * (1 + xi)) - np.log(0.5 * (1 + xi * xi)) + 2.0 * np.arctan(xi) - 0.5 * np.pi
        phi = (1.0 - 16.0 * x) ** -0.5
    absu = ustar / KAPPA * (np.log(z / z0) + psi)
    K = KAPPA * ustar * z / phi
    return z, (um / absum * absu, vm / absum * absu, K, K, K)


def _met(rng, zm, day=False):
    """Friction velocity, Obukhov length and wind vector of one half hour (``day``: of
    the unstable hours only; the default mode keeps the reference's rounding, which
    drowns a fine grid's footprint in stable hours)."""
    ustar = float(rng.uniform(0.28, 0.35))
    stable = rng.random() < 0.25 and not day
    mol = float(zm * rng.uniform(6.0, 12.0)) if stable else float(-zm * rng.uniform(2.0, 4.0))
    speed = ustar / KAPPA * (rng.uniform(5.0, 6.0) + _psi(zm / mol))
    th = rng.uniform(0.0, 2.0 * math.pi)
    return ustar, mol, (-speed * math.sin(th), -speed * math.cos(th))


def _source(rng, nx, ny, dx):
    """A patchy surface flux: a few Gaussian sources on a weak background."""
    x, y = np.arange(nx) * dx, np.arange(ny) * dx
    q = np.full((ny, nx), 0.05)
    for _ in range(3):
        cx, cy, s = rng.uniform(0.2, 0.8) * nx * dx, rng.uniform(0.2, 0.8) * ny * dx, rng.uniform(3.0, 8.0) * dx
        q += rng.uniform(0.5, 1.5) * np.exp(-((x[None, :] - cx) ** 2 + (y[:, None] - cy) ** 2) / (2 * s * s))
    return q


def _levels(n, nlev):
    return n if nlev == 1 else [int(round(v)) for v in np.linspace(0, n, nlev)]


def _kwargs(c, rng):
    """steady_state_transport_solver's arguments of one (tower, time)."""
    ustar, mol, wind = _met(rng, c["zm"], c.get("mode") == "fp64")
    z, prof = _profiles(c["n"], c["zm"], wind, ustar, mol)
    nx, ny, dx = c["nx"], c["ny"], c["dx"]
    src = np.zeros((ny, nx)) if c["footprint"] else _source(rng, nx, ny, dx)
    shift = c.get("shift", True)
    meas = (float(rng.uniform(0.3, 0.7)) * nx * dx, float(rng.uniform(0.3, 0.7)) * ny * dx) if shift else (0.0, 0.0)
    halo = c.get("halo", -1.0)
    return dict(srf_flx=src, z=z, profiles=prof, domain=(nx * dx, ny * dx), levels=_levels(c["n"], c["nlev"]),
                modes=(c["mx"], c["my"]), meas_pt=meas, footprint=c["footprint"], halo=None if halo < 0 else halo,
                precision=c.get("precision", "double"))


def _batch_kwargs(c, seed):
    rng = np.random.default_rng(seed)
    if c["nx"]:
        return [_kwargs(c, rng) for _ in range(c["count"])]
    out = []
    for k in range(c["count"]):
        grid, n, dom = TOWERS[k % len(TOWERS)]
        out.append(_kwargs(dict(nx=grid, ny=grid, dx=dom / grid, n=n, zm=float(rng.uniform(4.0, 8.0)) * dom / grid,
                                mx=grid, my=grid, nlev=1, footprint=True), rng))
    return out


def _surrogate_items(c, seed):
    """Met cases inside the n = 128 network's box."""
    rng = np.random.default_rng(seed)
    zm = min(20.0, 8.0 * c["dx"])
    out = []
    for _ in range(c["count"]):
        s1, s2 = float(rng.uniform(-0.9, 0.2)), float(rng.uniform(4.7, 7.3))
        U = float(rng.uniform(2.0, 8.0))
        th = float(rng.uniform(0.0, 2.0 * math.pi))
        out.append(dict(n=128, zm=zm, wind=(-U * math.sin(th), -U * math.cos(th)), srf_shape=(c["ny"], c["nx"]),
                        domain=(c["nx"] * c["dx"], c["ny"] * c["dx"]), modes=(_even(c["nx"]), _even(c["ny"])),
                        meas_pt=(0.5 * c["nx"] * c["dx"], 0.5 * c["ny"] * c["dx"]),
                        ustar=KAPPA * U / (s2 + _psi(s1)), mol=zm / s1))
    return out


def _series(c, seed):
    """vertical_profiles' arguments of every half hour of one tower."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(c["steps"]):
        ustar, mol, wind = _met(rng, c["zm"])
        out.append(dict(n=c["n"], meas_height=c["zm"], wind=wind, ustar=ustar, mol=mol))
    return out


def _series_kwargs(c, z, prof):
    lx, ly = c["nx"] * c["dx"], c["ny"] * c["dx"]
    return dict(srf_flx=_series_field(c["ny"], c["nx"]), z=z, profiles=prof, domain=(lx, ly), levels=c["n"],
                modes=(c["mx"], c["my"]), meas_pt=(0.5 * lx, 0.5 * ly), footprint=True, halo=None, precision="double")


@functools.lru_cache(maxsize=8)
def _series_field(ny, nx):
    return np.zeros((ny, nx))


def _train_inputs(c, seed):
    """Samples as the transfer pool gives them (features of (k, met case), smooth
    targets that decay with k, weights over several decades) and He-scaled weights."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    m = c["samples"]

    def u(lo, hi):
        return torch.rand(m, generator=g, device=DEV) * (hi - lo) + lo

    s1, s2, lk, th = u(-1.25, 0.35), u(4.25, 7.75), u(math.log(1e-3), math.log(40.0)), u(0.0, 0.5 * math.pi)
    k = lk.exp()
    kpar, kperp = k * th.cos(), k * th.sin()
    X = torch.stack([kpar / 10, kperp / 10, s1, (s2 - 6.0) / 1.5, 2.0 / s2 - 0.3, lk / 3, th.cos(), s1.clamp(min=0) * 4], 1)
    r = k / (1.0 + k)
    T = torch.stack([-r * (0.6 + 0.2 * s1), -r * th.cos() * 6.0 / s2, 0.3 * r * s1, 0.4 * r * th.cos()], 1)
    w = (k * k * torch.exp(-2.0 * k)).unsqueeze(1) * torch.tensor([20.0, 20.0, 8.0, 8.0], device=DEV) + 1e-3
    H = 256
    parts = [torch.randn(8 * H, generator=g, device=DEV) * math.sqrt(2.0 / 8), torch.zeros(H, device=DEV)]
    for _ in range(3):
        parts += [torch.randn(H * H, generator=g, device=DEV) * math.sqrt(2.0 / H), torch.zeros(H, device=DEV)]
    parts += [torch.randn(4 * H, generator=g, device=DEV) * math.sqrt(1.0 / H), torch.zeros(4, device=DEV)]
    return X.float().contiguous(), T.float().contiguous(), w.float().contiguous(), torch.cat(parts).float()


LR = 1e-5  # the last stretch of the training schedule


def _points_inputs(c, seed):
    """Footprints (positive, skewed, their sum near one) and flux maps."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    shape = (c["count"], c["ny"], c["nx"])
    F = torch.empty(shape, dtype=torch.float64, device=DEV).exponential_(1.0, generator=g) ** 2
    F /= 2.0 * c["nx"] * c["ny"]
    G = torch.randn(shape, dtype=torch.float64, generator=g, device=DEV) * 0.3 + 1.0
    return F, G


_SOLVERS = {}


def _solvers(c, count):
    """The batch solvers a serving program keeps for a workload (one, or several in
    flight), made once per workload and kept while the process runs."""
    from bldfm_gb300.batch import BatchSolver

    key = tuple(sorted((k, v) for k, v in c.items() if k != "name"))
    if key not in _SOLVERS:
        _SOLVERS[key] = [BatchSolver() for _ in range(count)]
    return _SOLVERS[key]


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        from bldfm_gb300 import steady_state_transport_solver

        return dict(kind=kind, f=steady_state_transport_solver, mode=c["mode"],
                    kw=_kwargs(c, np.random.default_rng(seed)))
    if kind in ("batch", "batch_host"):
        from bldfm_gb300.batch import solve_batch

        return dict(kind=kind, solver=_solvers(c, 1)[0], f=solve_batch, cases=_batch_kwargs(c, seed))
    if kind == "timeseries":
        from bldfm_gb300.batch import solve_stream
        from bldfm_gb300.pbl_model import vertical_profiles_batch

        return dict(kind=kind, profiles=vertical_profiles_batch, stream=solve_stream, solvers=_solvers(c, 3), c=c,
                    met=_series(c, seed))
    if kind == "surrogate":
        from bldfm_gb300 import surrogate as S

        net, box, _ = S.load(batch=256)
        sur = S.Surrogate(net, box=box)
        return dict(kind=kind, sur=sur, batch=sur.prepare_batch(_surrogate_items(c, seed)))
    if kind == "train":
        from bldfm_gb300.mlp import MLP

        X, T, w, p = _train_inputs(c, seed)
        net = MLP(batch=c["samples"])
        net.set_params(p.cpu().numpy())
        return dict(kind=kind, net=net, X=X, T=T, w=w)
    from bldfm_gb300.utils import point_measurement_batch

    F, G = _points_inputs(c, seed)
    return dict(kind=kind, f=point_measurement_batch, F=F, G=G)


def run(state):
    s, kind = state, state["kind"]
    if kind == "solve":
        _, conc, flx = s["f"](**s["kw"], mode=s["mode"])
        return [conc, flx]
    if kind == "batch":
        return [x for pair in s["solver"].solve(s["cases"]) for x in pair]
    if kind == "batch_host":
        return [x for _, conc, flx in s["f"](s["cases"], solver=s["solver"]) for x in (conc, flx)]
    if kind == "timeseries":
        cases = [_series_kwargs(s["c"], z, prof) for z, prof in s["profiles"](s["met"])]
        batches = [cases[k:k + 16] for k in range(0, len(cases), 16)]
        res = [r for b in s["stream"](batches, solvers=s["solvers"]) for r in b]
        return [np.stack([r[1] for r in res]), np.stack([r[2] for r in res])]
    if kind == "surrogate":
        return [x for pair in s["sur"].solve_batch_prepared(s["batch"]) for x in pair]
    if kind == "train":
        s["net"].train_step(s["X"], s["T"], s["w"], LR)
        grads, loss = s["net"].grads()
        return dict(grads=grads, loss=loss, params=s["net"].params())
    return s["f"](s["F"], s["G"])


# --------------------------------------------------------------------------- work


def _solve_work(nx, ny, halo_cells, mx, my, nz, jmax, nlev, footprint):
    """The invariant-imbedding sweep of half the modes (42 or 56 flops a step), the
    pruned transforms, and the fields in and out."""
    nxe, nye = nx + 2 * halo_cells, ny + 2 * halo_cells
    sweep = 0.5 * mx * my * (42.0 * (nz - 1 - jmax) + 56.0 * jmax)
    fft = 5.0 * nlev * (mx * nye * math.log2(nye) + ny * nxe * math.log2(nxe))
    byts = 16.0 * nx * ny * nlev
    if not footprint:
        fft += 2.5 * (ny * nxe * math.log2(nxe) + mx * nye * math.log2(nye))
        byts += 8.0 * nx * ny
    return byts, sweep + fft


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        n = c["samples"]
        # three hidden layers forward, data gradient and weight gradient; samples in, gradients and weights out
        return {"bytes": 64.0 * n + 8.0 * 200708, "flops": 2.0 * n * 9 * 256 * 256 + 6.0 * n * 12 * 256}
    if kind == "points":
        n = c["count"] * c["nx"] * c["ny"]
        return {"bytes": 16.0 * n + 8.0 * c["count"], "flops": 2.0 * n}
    if kind == "surrogate":
        b, f = _solve_work(c["nx"], c["ny"], max(c["nx"], c["ny"]), c["nx"], c["ny"], 1, 0, 1, True)
        modes = 0.5 * c["nx"] * c["ny"]
        return {"bytes": b * c["count"], "flops": (f + modes * 2.0 * 256 * (3 * 256 + 12)) * c["count"]}
    if kind == "timeseries":
        b, f = _solve_work(c["nx"], c["ny"], max(c["nx"], c["ny"]), c["mx"], c["my"], int(1.6 * c["n"]), c["n"], 1, True)
        return {"bytes": b * c["steps"], "flops": f * c["steps"]}
    if kind == "solve":
        cells = max(c["nx"], c["ny"]) if c["halo"] < 0 else int(c["halo"] / c["dx"])
        b, f = _solve_work(c["nx"], c["ny"], cells, c["mx"], c["my"], int(1.6 * c["n"]), c["n"], c["nlev"],
                           c["footprint"])
        return {"bytes": b, "flops": f}
    if not c["nx"]:
        got = [_solve_work(g, g, g, g, g, int(1.6 * n), n, 1, True)
               for g, n, _ in (TOWERS[k % len(TOWERS)] for k in range(c["count"]))]
        return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}
    b, f = _solve_work(c["nx"], c["ny"], max(c["nx"], c["ny"]), c["mx"], c["my"], int(1.6 * c["n"]), c["n"], c["nlev"],
                       c["footprint"])
    return {"bytes": b * c["count"], "flops": f * c["count"]}


# --------------------------------------------------------------------------- 64-bit values


def _exact_solve(srf_flx, z, profiles, domain, levels, modes, meas_pt, footprint, halo, precision):
    """The discrete boundary-value problem in complex128: invariant imbedding from
    the radiation condition downwards, then the inverse transform and the crop."""
    c128, f64 = torch.complex128, torch.float64
    u, v, Kx, Ky, Kz = (np.asarray(a, dtype=np.float64) for a in profiles)
    nz = len(z)
    dz = np.diff(z)
    ny, nx = srf_flx.shape
    (xmx, ymx), (xm, ym) = domain, meas_pt
    dx, dy = xmx / nx, ymx / ny
    halo = max(xmx, ymx) if halo is None else halo
    px, py = int(halo / dx), int(halo / dy)
    nxe, nye = nx + 2 * px, ny + 2 * py
    nlx, nly = modes
    if nlx > nxe or nly > nye:
        nlx, nly = nxe, nye
    dlx, dly = (nxe - nlx) // 2, (nye - nly) // 2
    if footprint:
        q0 = torch.full((nly, nlx), 1.0 / nxe / nye, dtype=c128, device=DEV)
    else:
        pad = torch.zeros((nye, nxe), dtype=c128, device=DEV)
        pad[py:py + ny, px:px + nx] = torch.as_tensor(srf_flx, device=DEV)
        f = torch.fft.fftshift(torch.fft.fft2(pad, norm="forward"))
        q0 = torch.fft.ifftshift(f[dly:nye - dly, dlx:nxe - dlx])
    lx = 2.0 * np.pi / dx / nxe * torch.fft.fftfreq(nlx, d=1.0 / nlx, dtype=f64, device=DEV)
    ly = 2.0 * np.pi / dy / nye * torch.fft.fftfreq(nly, d=1.0 / nly, dtype=f64, device=DEV)
    Lx, Ly = lx[None, :].expand(nly, nlx), ly[:, None].expand(nly, nlx)
    k = 1.0 / Kz[-1]
    eig = torch.sqrt(torch.complex(Kx[-1] * k * Lx**2 + Ky[-1] * k * Ly**2, u[-1] * k * Lx + v[-1] * k * Ly))
    eig[0, 0] = 1.0
    R = 1.0 / (Kz[-1] * eig)
    Q = torch.ones_like(R)  # product of the flux factors above the level, scaled
    logs = torch.zeros((nly, nlx), dtype=f64, device=DEV)
    want = [levels] if np.ndim(levels) == 0 else list(levels)
    kept = {}
    for i in range(nz - 2, -1, -1):
        if i + 1 in want:
            kept[i + 1] = (R.clone(), Q.clone(), logs.clone())
        K, h = 1.0 / Kz[i], dz[i]
        T = torch.complex(-(Kx[i] * Lx**2 + Ky[i] * Ly**2), -(u[i] * Lx + v[i] * Ly))
        a = 1.0 - 0.5 * K * h * h * T
        b = -K * h - K * K * h**3 / 6.0 * T
        cc = T * (h - K * h**3 / 6.0 * T)
        R = (a * R - b) / (a - cc * R)
        Q = Q * (cc * R + a)
        if i % 8 == 0:
            m = Q.abs().clamp(min=1e-290)
            Q, logs = Q / m, logs + m.log()
    if 0 in want:
        kept[0] = (R.clone(), Q.clone(), logs.clone())
    p00 = [0.0]
    for i in range(nz - 1):
        p00.append(p00[-1] - float(q0[0, 0].real) * dz[i] * (0.5 / Kz[i] + 0.5 / Kz[i + 1]))
    shift = None
    if footprint:
        shift = torch.exp(1j * (Lx * (xm + halo) + Ly * (ym + halo)))
    elif xm**2 + ym**2 > 0.0:
        shift = torch.exp(1j * (Lx * (xm - xmx / 2) + Ly * (ym - ymx / 2)))
    out = ([], [])
    for j in sorted(set(want)):
        Rj, Qj, lj = kept[j]
        q = q0 * (Q / Qj) * torch.exp(logs - lj)
        p = Rj * q
        q[0, 0], p[0, 0] = q0[0, 0], p00[j]
        for spec, to in ((p, out[0]), (q, out[1])):
            spec = spec if shift is None else spec * shift
            full = torch.nn.functional.pad(torch.fft.fftshift(spec), (dlx, dlx, dly, dly))
            full = torch.fft.ifftshift(full)
            fld = torch.fft.fft2(full).real if footprint else torch.fft.ifft2(full, norm="forward").real
            to.append(fld[py:nye - py, px:nxe - px])
    return tuple(torch.stack(o) for o in out)


def _dropin_exact(kw):
    conc, flx = _exact_solve(**kw)
    conc, flx = conc.squeeze(), flx.squeeze()
    return [conc, flx]


def _mlp_exact(X, T, w, p):
    """Gradients, loss and first Adam update of the network in FP64."""
    X, T, w, p = (t.double() for t in (X, T, w, p))
    H, o, parts = 256, 0, []
    for shape in [(8, H), (H,)] + [(H, H), (H,)] * 3 + [(H, 4), (4,)]:
        size = int(np.prod(shape))
        parts.append(p[o:o + size].reshape(shape).clone().requires_grad_(True))
        o += size
    gelu = functools.partial(torch.nn.functional.gelu, approximate="tanh")
    h = gelu(X @ parts[0] + parts[1])
    for j in range(3):
        h = gelu(h @ parts[2 + 2 * j].T + parts[3 + 2 * j])
    loss = (w * (h @ parts[8] + parts[9] - T) ** 2).sum() / X.shape[0]
    g = torch.cat([t.reshape(-1) for t in torch.autograd.grad(loss, parts)])
    return dict(grads=g, loss=loss.detach(), params=p - LR * g / (g.abs() + 1e-8))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        return _dropin_exact(_kwargs(c, np.random.default_rng(seed)))
    if kind in ("batch", "batch_host"):
        host = kind == "batch_host"
        out = []
        for kw in _batch_kwargs(c, seed):
            pair = _exact_solve(**kw)
            out += [t.squeeze() for t in pair] if host else list(pair)
        return out
    if kind == "timeseries":
        out = ([], [])
        for m in _series(c, seed):
            z, prof = _profiles(m["n"], m["meas_height"], m["wind"], m["ustar"], m["mol"])
            for t, to in zip(_exact_solve(**_series_kwargs(c, z, prof)), out):
                to.append(t.squeeze())
        return [torch.stack(o) for o in out]
    if kind == "surrogate":
        out = []
        for it in _surrogate_items(c, seed):
            z, prof = _profiles(it["n"], it["zm"], it["wind"], it["ustar"], it["mol"])
            pair = _exact_solve(np.zeros(it["srf_shape"]), z, prof, it["domain"], it["n"], it["modes"], it["meas_pt"],
                                True, None, "single")
            out += [t.squeeze() for t in pair]
        return out
    if kind == "train":
        return _mlp_exact(*_train_inputs(c, seed))
    F, G = _points_inputs(c, seed)
    F, G = F.reshape(c["count"], -1), G.reshape(c["count"], -1)
    return (F * G).sum(1)
