"""Performance cases: the work a user of pyexner_b200 has it do, through its public entry points.

A pass restarts from the initial state it holds and takes a fixed number of steps (or runs to
a fixed time), as a program that makes a run, a parameter study or a gradient does:

* ``bed``      Roe-Exner on a rectangular grid with ring boundaries (the fused stage path):
               ``init_fn`` and ``run_steps``; optionally with nodata holes (islands).
* ``ldomain``  Roe-Exner on an L-shaped domain: NaN-bed block, walls inside the array, an
               inflow (the general stage path).
* ``berthon``  the analytic erosion channel through the time-driven integrator loop with
               output windows and time-dependent handlers (one host decision per step).
* ``ensemble`` a ragged ensemble of dam breaks, all members advanced together.
* ``roe``      the plain Roe dam break.
* ``vjp``      gradient of a bed misfit with respect to the initial state, the inflow
               discharge and the sediment matrix (forward run, backward sweep, init).
* ``jvp``      directional derivative of a run.

``exact`` is the same mathematics in plain torch on float64 (PyExner's formulas), gradients by
torch's own differentiation.
"""
import functools
import math

import numpy as np
import torch
import torch.autograd.forward_ad as fwAD

import pyexner_b200 as pe
from pyexner_b200 import cases as workloads
from pyexner_b200.boundaries import BoundaryManager, index_coords, ring_boundaries
from pyexner_b200.ensemble import Ensemble
from pyexner_b200.integrators import scratch_like
from pyexner_b200.tangent import ParamAdjoints, jvp_init, jvp_run, vjp_init, vjp_run

CFL = 0.5
DX = 0.01


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference's erosion channel input (71 x 12 cells) run to a time: the smallest grid,
        # every step decided on the host; what a first run of the framework looks like
        dict(name="berthon_71x12", kind="berthon", dh=0.1, dtype="float32", end_time=0.4, out_freq=0.2),
        # a small grid, fixed step count: latency and launches count
        dict(name="bed_100x96", kind="bed", ny=96, nx=100, dtype="float32", scheme="SSPRK2", steps=100, u0=0.1,
             grass="MPM", nsed=1, inflow=False, holes=0),
        # the headline workload: Gaussian bed at 2048^2, started below the bedload threshold
        dict(name="bed_2048", kind="bed", ny=2048, nx=2048, dtype="float32", scheme="SSPRK2", steps=20, u0=0.1,
             grass="MPM", nsed=1, inflow=False, holes=0),
        # the same grid with bedload in every cell
        dict(name="transport_2048", kind="bed", ny=2048, nx=2048, dtype="float32", scheme="SSPRK2", steps=20, u0=1.0,
             grass="MPM", nsed=1, inflow=False, holes=0),
        # the bandwidth workload: the largest grid
        dict(name="bed_8192", kind="bed", ny=8192, nx=8192, dtype="float32", scheme="SSPRK2", steps=8, u0=0.1,
             grass="MPM", nsed=1, inflow=False, holes=0),
        # float64, as used for accuracy checks and as the base of the derivatives
        dict(name="bed_1024_f64", kind="bed", ny=1024, nx=1024, dtype="float64", scheme="SSPRK2", steps=20, u0=1.0,
             grass="MPM", nsed=1, inflow=False, holes=0),
        # an ordinary odd-sized river reach with islands, an inflow, a constant grass factor, Forward Euler
        dict(name="islands_731x1203", kind="bed", ny=731, nx=1203, dtype="float32", scheme="FE", steps=41, u0=0.6,
             grass="0.005", nsed=1, inflow=True, holes=6),
        # an irregular domain with inner walls
        dict(name="ldomain_503x701", kind="ldomain", ny=503, nx=701, dtype="float32", scheme="SSPRK2", steps=20, u0=0.6,
             grass="MPM"),
        # the plain shallow-water solver, the reference's dam break configuration
        dict(name="roe_256_f64", kind="roe", ny=256, nx=256, dtype="float64", scheme="SSPRK2", steps=200),
        # many independent grids of different sizes
        dict(name="ensemble_24", kind="ensemble", count=24, lo=128, hi=640, dtype="float32", scheme="SSPRK2", steps=40),
        # gradients of the 512^2 inflow case
        dict(name="vjp_512", kind="vjp", ny=512, nx=512, scheme="SSPRK2", steps=16, every=8),
        # a directional derivative
        dict(name="jvp_256", kind="jvp", ny=256, nx=256, scheme="SSPRK2", steps=12),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("bed", "bed", "bed", "bed", "ldomain", "berthon", "roe", "ensemble", "vjp", "jvp"))
    scheme = rng.choice(("SSPRK2", "SSPRK2", "FE"))
    if kind == "bed":
        dtype = rng.choice(("float32", "float32", "float64"))
        top = 5000 if dtype == "float32" else 1500
        ny, nx = log(48, top), log(48, top)
        steps = max(4, min(100, int(6e7 / (ny * nx)), 10 + rng.randrange(60)))
        return dict(kind=kind, ny=ny, nx=nx, dtype=dtype, scheme=scheme, steps=steps, u0=rng.choice((0.1, 1.0)),
                    grass=rng.choice(("MPM", "MPM", "0.005")), nsed=rng.choice((1, 1, 2)),
                    inflow=rng.random() < 0.3, holes=rng.choice((0, 0, 3)))
    if kind == "ldomain":
        return dict(kind=kind, ny=log(40, 900), nx=log(40, 900), dtype=rng.choice(("float32", "float64")),
                    scheme=scheme, steps=8 + rng.randrange(12), u0=rng.choice((0.1, 0.9)),
                    grass=rng.choice(("MPM", "0.005")))
    if kind == "berthon":
        return dict(kind=kind, dh=0.2 / rng.randrange(1, 7), dtype=rng.choice(("float32", "float64")),
                    end_time=0.1 + 0.05 * rng.randrange(4), out_freq=rng.choice((0.05, 0.2)))
    if kind == "roe":
        return dict(kind=kind, ny=log(40, 700), nx=log(40, 700), dtype=rng.choice(("float64", "float64", "float32")),
                    scheme=scheme, steps=20 + rng.randrange(100))
    if kind == "ensemble":
        return dict(kind=kind, count=4 + rng.randrange(20), lo=64, hi=200 + rng.randrange(400),
                    dtype=rng.choice(("float32", "float32", "float64")), scheme=scheme, steps=6 + rng.randrange(20))
    if kind == "vjp":
        return dict(kind=kind, ny=log(40, 480), nx=log(40, 480), scheme=scheme, steps=4 + rng.randrange(12),
                    every=rng.choice((4, 8, 32)))
    return dict(kind="jvp", ny=log(40, 300), nx=log(40, 300), scheme=scheme, steps=3 + rng.randrange(9))


# ------------------------------------------------------------------------------ inputs
def _dtype(case):
    return torch.float32 if case.get("dtype", "float64") == "float32" else torch.float64


def _bed(gen, ny, nx, dx=DX, scale=0.05, modes=16):
    """Sum of Gaussian bumps on the (ny + 2) x (nx + 2) grid, float64 on the GPU."""
    lx, ly = nx * dx, ny * dx
    side = math.sqrt(lx * ly)
    r = torch.rand((4, modes), generator=gen, dtype=torch.float64).tolist()
    x = (torch.arange(nx + 2, dtype=torch.float64, device="cuda") - 0.5) * dx
    y = (ny + 1 - torch.arange(ny + 2, dtype=torch.float64, device="cuda") - 0.5) * dx
    rows, cols = [], []
    for a, b, s, w in zip(*r):
        s = (0.05 + 0.25 * s) * side
        rows.append((2 * w - 1) * torch.exp(-((y - b * ly) ** 2) / (2 * s * s)))
        cols.append(torch.exp(-((x - a * lx) ** 2) / (2 * s * s)))
    return scale * torch.stack(rows, 1) @ torch.stack(cols, 0)


def _noise(gen, shape):
    """Uniform in (-1, 1) on the GPU, from the seed of `gen`."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(torch.randint(0, 2**62, (1,), generator=gen)))
    return 2.0 * torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") - 1.0


def _channel(gen, ny, nx, u0):
    """Still-surface water with 2 % noise over an erodible Gaussian bed, moving at u0 in x."""
    zt = _bed(gen, ny, nx)
    z = torch.full_like(zt, float(zt.min()) - 0.05)
    h = ((0.3 - zt) * (1.0 + 0.02 * _noise(gen, zt.shape))).clamp_min(0.0)
    zero = torch.zeros_like(zt)
    return dict(h=h, hu=u0 * h, hv=zero, z=z, z_b=zt - z, n=zero, G=zero)


def _seds(nsed):
    """7 x nsed sediment matrix: fraction, d50, density, deposition, erosion, theta_c, porosity."""
    if nsed == 1:
        return np.array([[1.0], [1.61e-3], [2630.0], [0.0], [0.0], [0.047], [0.42]])
    return np.array([[0.6, 0.4], [1.61e-3, 0.9e-3], [2630.0, 2650.0], [0.0, 0.0], [0.0, 0.0], [0.047, 0.047], [0.42, 0.42]])


def _erosion(case):
    if case.get("grass", "MPM") != "MPM":
        return dict(grass_factor=float(case["grass"]))
    m = _seds(case.get("nsed", 1))
    seds = {"s%d" % k: dict(fraction=m[0, k], diameter=m[1, k], density=m[2, k], deposition_flux=0.0, erosion_flux=0.0)
            for k in range(m.shape[1])}
    return dict(grass_factor="MPM", bulk_porosity=0.42, sediments=seds)


def _rect(x0, x1, y0, y1):
    return [[x0 - 0.5, y0 - 0.5], [x1 + 0.5, y0 - 0.5], [x1 + 0.5, y1 + 0.5], [x0 - 0.5, y1 + 0.5]]


def _block(ny, nx):
    """Rows and columns of the L-shaped domain's missing corner (top right)."""
    return max(4, (ny + 2) // 3), max(4, (nx + 2) // 3)


@functools.lru_cache(maxsize=64)
def _layout(kind, ny, nx, inflow=False):
    """The boundary handlers of a grid, which depend on its shape alone."""
    gy, gx = ny + 2, nx + 2
    if kind == "roe":
        spec = ring_boundaries(gy, gx, ["Reflective"], ["Reflective"], ["Reflective"], ["Reflective"])
    elif kind == "ldomain":
        br, bc = _block(ny, nx)
        c0 = gx - bc  # first column of the block

        def e(t, poly, normal, values=(0.0, 0.0, 0.0, 0.0)):
            return {"type": t, "polygon": poly, "values": list(values), "normal": normal}

        spec = {
            "inlet": e("ConstantInflux", _rect(0, 0, 0, gy - 1), [-1.0, 0.0], (0.18, 1.0, 0.0, 0.0)),
            "inlet_bed": e("TransmissiveBed", _rect(0, 0, 0, gy - 1), [-1.0, 0.0]),
            "outlet": e("Transmissive", _rect(gx - 1, gx - 1, 0, gy - 1 - br), [1.0, 0.0]),
            "outlet_bed": e("TransmissiveBed", _rect(gx - 1, gx - 1, 0, gy - 1 - br), [1.0, 0.0]),
            "wall": e("Reflective", _rect(c0 - 1, c0 - 1, gy - br, gy - 1), [1.0, 0.0]),
            "ceiling": e("Reflective", _rect(c0, gx - 2, gy - br - 1, gy - br - 1), [0.0, 1.0]),
            "bottom": e("Reflective", _rect(0, gx - 1, 0, 0), [0.0, -1.0]),
            "top": e("Reflective", _rect(0, c0 - 1, gy - 1, gy - 1), [0.0, 1.0]),
        }
    else:
        west = [("ConstantInflux", [0.3, 1.0, 0.0, 0.0]), "TransmissiveBed"] if inflow else ["Transmissive", "TransmissiveBed"]
        spec = ring_boundaries(gy, gx, west, ["Transmissive", "TransmissiveBed"], ["Reflective"], ["Reflective"])
    X, Y = index_coords(gy, gx)
    scheme = "Roe" if kind == "roe" else "Roe Exner"
    return BoundaryManager(dict(flux_scheme=scheme, boundaries=spec), X, Y, setup="device")


def _arrays(case, seed):
    """The initial planes of a single-grid case, float64 on the GPU."""
    gen = torch.Generator()
    gen.manual_seed(int(seed))
    kind, ny, nx = case["kind"], case["ny"], case["nx"]
    if kind == "roe":
        r = torch.rand(3, generator=gen, dtype=torch.float64).tolist()
        h = torch.empty((ny + 2, nx + 2), dtype=torch.float64, device="cuda")
        cut = int((0.4 + 0.2 * r[0]) * (nx + 2))
        h[:, :cut] = 0.8 + 0.4 * r[1]
        h[:, cut:] = 0.1 + 0.1 * r[2]
        h *= 1.0 + 0.01 * _noise(gen, h.shape)
        zero = torch.zeros_like(h)
        return dict(h=h, hu=zero, hv=zero, z=zero, n=zero)
    a = _channel(gen, ny, nx, case.get("u0", 1.0))
    if kind == "bed" and case["grass"] != "MPM" or kind == "ldomain" and case["grass"] != "MPM":
        a["G"] = torch.full_like(a["h"], float(case["grass"]))
    if kind == "ldomain":
        br, bc = _block(ny, nx)
        a["z"] = a["z"].clone()
        a["z"][:br, nx + 2 - bc:] = float("nan")
    if kind == "bed" and case["holes"]:
        a["z"] = a["z"].clone()
        r = torch.rand((case["holes"], 4), generator=gen, dtype=torch.float64).tolist()
        for x, y, p, q in r:
            i, j = int(2 + y * (ny - 8)), int(2 + x * (nx - 8))
            a["z"][i:min(ny, i + 2 + int(p * 0.1 * ny)), j:min(nx, j + 2 + int(q * 0.1 * nx))] = float("nan")
    return a


def _fill(state, arrs):
    for f, v in arrs.items():
        getattr(state, f).copy_(v)
    return state


def _berthon(case, seed):
    x, y, fields, params = workloads.berthon_case(dh=case["dh"], end_time=case["end_time"], out_freq=case["out_freq"])
    rng = np.random.default_rng(seed)
    fields = dict(fields)
    fields["h"] = fields["h"] * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, fields["h"].shape))
    fields["G"] = np.full(fields["h"].shape, 0.005)
    return x, y, fields, params


def _members(case, seed):
    """(shape, planes) of every member: dam breaks over their own beds, at rest."""
    gen = torch.Generator()
    gen.manual_seed(int(seed))
    sizes = torch.Generator()
    sizes.manual_seed(20 + case["count"])
    out = []
    for _ in range(case["count"]):
        ny, nx = torch.randint(case["lo"], case["hi"] + 1, (2,), generator=sizes).tolist()
        zt = _bed(gen, ny, nx)
        z = torch.full_like(zt, float(zt.min()) - 0.05)
        h = (0.3 - zt).clamp_min(0.0)
        h[:, : (nx + 2) // 2] += 0.2 + 0.8 * float(torch.rand((), generator=gen, dtype=torch.float64))
        zero = torch.zeros_like(zt)
        out.append(((ny, nx), dict(h=h, hu=zero, hv=zero, z=z, z_b=zt - z, n=zero, G=zero)))
    return out


def _target(case, seed):
    gen = torch.Generator()
    gen.manual_seed(int(seed) + 1_000_003)
    return _bed(gen, case["ny"], case["nx"])


def _direction(case, seed):
    gen = torch.Generator()
    gen.manual_seed(int(seed) + 2_000_003)
    shape = (case["ny"] + 2, case["nx"] + 2)
    return {f: s * _noise(gen, shape) for f, s in (("h", 0.01), ("hu", 0.01), ("hv", 0.01), ("z_b", 0.01))}


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "berthon":
        x, y, fields, params = _berthon(case, seed)
        X, Y = np.meshgrid(x, y, indexing="xy")
        bounds = BoundaryManager(params, X, Y)
        state = pe.RoeExnerState.from_numpy(fields, np.zeros((1, 1)), dtype=case["dtype"])
        solver, integ = pe.create_solver_bundle("Roe Exner"), pe.create_integrator_bundle("Forward Euler")
        cfg = solver.config(state, None, bounds, case["dh"], params)
        s.update(state=state, integ=integ, mask=bounds.boundary_mask,
                 config=integ.config(CFL, case["end_time"], case["out_freq"], solver, cfg))
        return s
    if kind == "ensemble":
        erosion = _erosion(case)
        members, start, live = [], [], []
        for (ny, nx), arrs in _members(case, seed):
            state = _fill(pe.RoeExnerState.empty((ny + 2, nx + 2), dtype=_dtype(case), seds=_seds(1)), arrs)
            members.append(dict(state=state, boundaries=_layout("bed", ny, nx), dx=DX))
            live += [getattr(state, f) for f in ("h", "hu", "hv", "z_b", "G")]
        start = [t.clone() for t in live]
        ens = Ensemble(members, erosion, dtype=_dtype(case))
        s.update(ens=ens, live=live, start=start)
        return s
    arrs = _arrays(case, seed)
    ny, nx = case["ny"], case["nx"]
    if kind == "roe":
        state = _fill(pe.RoeState.empty((ny + 2, nx + 2), dtype=_dtype(case)), arrs)
        solver = pe.create_solver_bundle("Roe")
        cfg = solver.config(state, None, _layout("roe", ny, nx), 1.0 / 256, {})
        s.update(state=state, solver=solver, cfg=cfg, mask=solver.mask_fn(state), scratch=scratch_like(state))
        return s
    state = _fill(pe.RoeExnerState.empty((ny + 2, nx + 2), dtype=_dtype(case), seds=_seds(case.get("nsed", 1))), arrs)
    bounds = _layout("ldomain" if kind == "ldomain" else "bed", ny, nx, kind == "vjp" or bool(case.get("inflow")))
    solver = pe.create_solver_bundle("Roe Exner")
    cfg = solver.config(state, None, bounds, DX, dict(erosion=_erosion(case)))
    s.update(state=state, solver=solver, cfg=cfg, mask=solver.mask_fn(state, None, bounds.boundary_mask),
             scratch=scratch_like(state))
    if kind == "vjp":
        s["target"] = _target(case, seed)
    if kind == "jvp":
        s["dot"] = _fill(pe.RoeExnerState.empty((ny + 2, nx + 2), dtype=torch.float64, seds=state.seds),
                         dict(_direction(case, seed), z=torch.zeros_like(arrs["h"])))
    return s


# ------------------------------------------------------------------------------ one pass
FIELDS = ("h", "hu", "hv", "z_b", "n_b", "G")


def _planes(state, fields=FIELDS):
    return {f: getattr(state, f) for f in fields}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "berthon":
        return _planes(s["integ"].run_fn(s["state"], s["config"], b_mask=s["mask"]))
    if kind == "ensemble":
        torch._foreach_copy_(s["live"], s["start"])
        s["ens"].init()
        dts = s["ens"].run(case["steps"], case["scheme"], cfl=CFL)
        out = [m["state"] for m in s["ens"].members]
        return dict(dts=dts, first=_planes(out[0]), last=_planes(out[-1]), h=[st.h for st in out[1:-1]],
                    z_b=[st.z_b for st in out[1:-1]])
    state, mask, cfg = s["state"], s["mask"], s["cfg"]
    if kind == "jvp":
        st, dot = jvp_init(state, s["dot"], mask, cfg)
        dts, dts_dot = jvp_run(st, dot, mask, cfg, case["steps"], case["scheme"], CFL)
        return dict(value=_planes(st), dot=_planes(dot, ("h", "hu", "hv", "z_b", "G")), dts=dts, dts_dot=dts_dot)
    st = s["solver"].init_fn(state, mask, cfg)
    if kind != "vjp":
        dts = pe.run_steps(st, mask, cfg, case["scheme"], case["steps"], CFL, scratch=s["scratch"])
        return dict(_planes(st, ("h", "hu", "hv", "z", "n") if kind == "roe" else FIELDS), dts=dts)
    end = st.clone()
    pe.run_steps(end, mask, cfg, case["scheme"], case["steps"], CFL, scratch=s["scratch"])
    bar = pe.RoeExnerState.empty(state.shape, dtype=torch.float64, seds=state.seds)
    bar.z.zero_()
    misfit = end.z + end.z_b - s["target"]
    bar.z_b.copy_(2.0 * misfit)
    params = ParamAdjoints(cfg, state.seds)
    vjp_run(st, bar, mask, cfg, case["steps"], case["scheme"], CFL, checkpoint_every=case["every"], params=params)
    vjp_init(state, bar, mask, cfg, params=params)
    return dict(cost=(misfit * misfit).sum(), grad=_planes(bar, ("h", "hu", "hv", "z_b")), d50=params.seds_bar[1],
                inflow=sum(params.inflow_bar.values()))


def work(case):
    """What a pass cannot do without: every step reads the state (h, hu, hv, z_b, G) and the
    static planes (z, n_b) once and writes the state once; a derivative pass also carries
    the state's derivatives.  Operations: about 650 per cell and stage of the Roe-Exner step
    (350 plain Roe), twice that again for a tangent, three times for an adjoint with its
    recomputed forward step."""
    kind = case["kind"]
    word = 4 if case.get("dtype", "float64") == "float32" else 8
    if kind == "berthon":
        cells = (7.0 / case["dh"]) * (1.0 / case["dh"] + 1)
        steps = case["end_time"] / (0.5 * case["dh"] / 5.5)
    elif kind == "ensemble":
        sizes = torch.Generator()
        sizes.manual_seed(20 + case["count"])
        cells = 0
        for _ in range(case["count"]):
            ny, nx = torch.randint(case["lo"], case["hi"] + 1, (2,), generator=sizes).tolist()
            cells += ny * nx
        steps = case["steps"]
    else:
        cells, steps = case["ny"] * case["nx"], case["steps"]
    stages = 2 if case.get("scheme") == "SSPRK2" else 1
    words = {"roe": 8, "jvp": 24, "vjp": 12 + 12 + 10}.get(kind, 12)
    ops = {"roe": 350, "jvp": 3 * 650, "vjp": 5 * 650}.get(kind, 650)
    return {"bytes": float(words * word * cells * steps), "flops": float(ops * cells * stages * steps)}


# ------------------------------------------------------------------------------ 64-bit answer
G_ACC, DRY, SED, VEL = 9.81, 1e-4, 1e-5, 1e-6


def _root(x):
    """Square root whose derivative is 0 at 0."""
    p = x > 0
    return torch.where(p, torch.sqrt(torch.where(p, x, torch.ones_like(x))), torch.zeros_like(x))


def _sides(t, axis):
    return (t[:, :-1], t[:, 1:]) if axis else (t[:-1], t[1:])


def _div(a, b, ok):
    return torch.where(ok, a / torch.where(ok, b, torch.ones_like(b)), torch.zeros_like(a))


def _spread(minus, plus, axis):
    """Cell sums of face values: `minus` to the first cell of each face, `plus` to the second."""
    pad = (lambda t, lo, hi: torch.nn.functional.pad(t, (lo, hi, 0, 0))) if axis else (
        lambda t, lo, hi: torch.nn.functional.pad(t, (0, 0, lo, hi)))
    return pad(minus, 0, 1) + pad(plus, 1, 0)


def _split(lams, alphas, betas, ents, ct, vt, force=None):
    pos, neg = [0.0, 0.0, 0.0], [0.0, 0.0, 0.0]
    zero = torch.zeros_like(ct)
    cols = ((1.0, lams[0], vt), (0.0, 0.0, ct), (1.0, lams[2], vt))
    for k in range(3):
        w = lams[k] * alphas[k] - betas[k]
        up, down = lams[k] > 0, lams[k] <= 0
        if force is not None:  # (all to the second cell, all to the first cell)
            up, down = (up | force[0]) & ~force[1], (down & ~force[0]) | force[1]
        e = ents[k] * alphas[k]
        for m in range(3):
            f, g = w * cols[k][m], e * cols[k][m]
            pos[m] = pos[m] + torch.where(up, f, zero) + torch.where(ents[k] > 0, g, zero)
            neg[m] = neg[m] + torch.where(down, f, zero) + torch.where(ents[k] < 0, g, zero)
    return pos, neg


def _exner_hydro(S, dt, dx, nod):
    """Roe-Exner hydrodynamic update: new h, hu, hv."""
    hc = S["h"].clamp_min(DRY)
    wet = hc > DRY
    u, v = _div(S["hu"], hc, wet), _div(S["hv"], hc, wet)
    bed = S["z"] + torch.where(S["z_b"] > SED, S["z_b"], torch.full_like(hc, SED * 0.01))
    bed = torch.where(nod, torch.zeros_like(bed), bed)
    flux = [0.0, 0.0, 0.0]
    for axis in (1, 0):
        n, t = (u, v) if axis else (-v, u)
        (hi, hj), (ui, uj), (vi, vj), (zi, zj) = (_sides(q, axis) for q in (hc, n, t, bed))
        si, sj = torch.sqrt(hi), torch.sqrt(hj)
        ht = 0.5 * (hi + hj)
        ct = torch.sqrt(G_ACC * ht)
        ut, vt = (ui * si + uj * sj) / (si + sj), (vi * si + vj * sj) / (si + sj)
        lams, ents, raw = [ut - ct, ut, ut + ct], [torch.zeros_like(ut)] * 3, (ut - ct, ut + ct)
        for k, sign, guard in ((0, -1.0, 0.0), (2, 1.0, VEL)):
            ei, ej = ui + sign * torch.sqrt(G_ACC * hi), uj + sign * torch.sqrt(G_ACC * hj)
            fix = (ei < 0) & (ej > 0)
            num = ei * (ej - lams[k]) if k == 0 else ej * (lams[k] - ei)
            ents[k] = torch.where(fix, lams[k] - _div(num, ej - ei, fix), torch.zeros_like(ut))
            lams[k] = torch.where(fix, _div(num, ej - ei + guard, fix), lams[k])
        dh, dq, dr = hj - hi, hj * uj - hi * ui, hj * vj - hi * vi
        alphas = ((-raw[1] * dh + dq) / (-2 * ct), (dr - vt * dh) / ct, (raw[0] * dh - dq) / (-2 * ct))
        nb = sum(_sides(S["n_b"], axis)) * 0.5
        slope = nb * nb * _root(ut * ut + vt * vt) * ut / (ht ** (4.0 / 3.0)).clamp_min(DRY)
        beta = (-G_ACC * ht * (zj - zi) - G_ACC * ht * slope * dx) / (-2 * ct)
        P, M = _split(lams, alphas, (beta, 0.0, -beta), ents, ct, vt)
        (di, dj), (mi, mj) = _sides(S["h"] > DRY, axis), _sides(nod, axis)
        on = (di | dj) & ~(mi | mj)
        P, M = ([torch.where(on, q, torch.zeros_like(q)) for q in R] for R in (P, M))
        if not axis:
            P, M = (P[0], P[2], -P[1]), (M[0], M[2], -M[1])
        flux = [f + _spread(m, p, axis) for f, m, p in zip(flux, M, P)]
    return [S[f] - dt * q / dx for f, q in zip(("h", "hu", "hv"), flux)]


def _corrections(h, hu, hv, ztot, nod):
    c = h[1:-1, 1:-1] + ztot[1:-1, 1:-1]

    def blocked(rows, cols):
        return ((c < ztot[rows, cols]) & (h[rows, cols] < DRY)) | nod[rows, cols]

    mid = slice(1, -1)
    live = (h[mid, mid] > DRY) & ~nod[mid, mid]
    ku = torch.ones_like(nod)
    kv = torch.ones_like(nod)
    ku[mid, mid] = live & ~blocked(mid, slice(2, None)) & ~blocked(mid, slice(0, -2))
    kv[mid, mid] = live & ~blocked(slice(0, -2), mid) & ~blocked(slice(2, None), mid)
    return torch.where(ku, hu, torch.zeros_like(hu)), torch.where(kv, hv, torch.zeros_like(hv))


def _grass(S, par, nod):
    if not par["mpm"]:
        g = S["G"]
        return torch.where((S["h"] > DRY) & ~nod, g, torch.zeros_like(g))
    h = S["h"].clamp_min(DRY)
    u, v = S["hu"] / h, S["hv"] / h
    m = par["seds"]
    total = 0.0
    for k in range(m.shape[1]):
        s1 = m[2, k] / 1000.0 - 1.0
        rough = m[1, k] ** (1.0 / 6.0) / 21.1
        theta = rough * rough * (u * u + v * v) / (s1 * m[1, k] * h ** (1.0 / 3.0))
        over = (theta - m[5, k]).clamp_min(0.0)
        total = total + m[0, k] * rough**3 * math.sqrt(G_ACC) / (s1 * torch.sqrt(h)) * 8.0 * _root(over) * over / (
            theta * _root(theta) + 1e-5)
    g = total / (1.0 - m[6].mean())
    return torch.where((S["h"] > DRY) & ~nod, g, torch.zeros_like(g))


def _exner_bed(S, dt, dx, nod):
    wet = S["h"] > DRY
    one = torch.ones_like(S["h"])
    h = torch.where(wet, S["h"], one * DRY * 0.01)
    u, v = _div(S["hu"], h, wet), _div(S["hv"], h, wet)
    zb = torch.where(S["z_b"] > SED, S["z_b"], one * SED * 0.01)
    sq, speed = torch.sqrt(h), u * u + v * v
    total = 0.0
    for axis in (1, 0):
        n = u if axis else -v
        (ni, nj), (si, sj), (ei, ej), (zi, zj) = (_sides(q, axis) for q in (n, sq, speed, zb))
        g = 0.5 * sum(_sides(S["G"], axis))
        qi, qj = g * ei * ni, g * ej * nj
        dz, dq, ut = zj - zi, qj - qi, ni * si + nj * sj
        big = dz.abs() > SED
        up = torch.where(big, _div(dq, dz, big), ut) >= 0
        (wi, wj), (mi, mj), (bi, bj) = _sides(wet, axis), _sides(nod, axis), _sides(S["z_b"] < SED, axis)
        on = (wi | wj) & ~(mi | mj) & ~(bi & bj)
        f = torch.where(on, torch.where(up, qi, qj), torch.zeros_like(qi))
        total = total + _spread(f, -f, axis)
    return S["z_b"] - dt * total / dx


def _handlers(S, par, time, scheme="exner"):
    for hd in par["handlers"]:
        kind, (b, d) = hd["kind"], hd["cells"]
        nx, ny = hd["normal"]
        v = hd["values"]
        shape = S["h"].shape
        new = {}

        def donor(f):
            return S[f].reshape(-1)[d]

        if kind == "Roe Exner Reflective":
            mn, mt = donor("hu") * nx + donor("hv") * ny, -donor("hu") * ny + donor("hv") * nx
            new = {f: donor(f) for f in ("h", "z_b", "n", "G")}
            new.update(hu=-mn * nx - mt * ny, hv=-mn * ny + mt * nx)
        elif kind == "Roe Exner Transmissive":
            new = {f: donor(f) for f in ("h", "hu", "hv")}
        elif kind == "Roe Exner TransmissiveBed":
            new = dict(z_b=donor("z_b"))
        elif kind == "Roe Exner ConstantInflux":
            q = par["q"].get(hd["name"], float(v[0]))
            new = dict(hu=q * float(v[1]), hv=q * float(v[2]))
        elif kind in ("Roe Exner Berthon", "Roe Exner NormalFlowDepth"):
            q, A, alpha, beta, gamma, x = (np.float32(w) for w in v[:6])
            w = np.float32(float((alpha * x + beta) / A) ** float(np.float32(1.0 / 3.0)))
            g2 = np.float32(2.0 * G_ACC)
            z0 = -(w * (w * w) + g2 * q) / (g2 * w) + gamma
            new = dict(z_b=float(-alpha * np.float32(time) + z0))
            if kind.endswith("Depth"):
                new.update(h=float(q / w), hu=donor("hu"), hv=donor("hv"))
        elif kind == "Roe Reflective":
            new = {f: donor(f) for f in ("h", "z", "n")}
            new.update(hu=donor("hu") * (1 - 2 * nx * nx), hv=donor("hv") * (1 - 2 * ny * ny))
        else:
            raise KeyError(kind)
        S = dict(S)
        for f, val in new.items():
            if not torch.is_tensor(val):
                val = torch.tensor(val, dtype=torch.float64, device="cuda")
            S[f] = S[f].reshape(-1).index_put((b,), val.expand(b.shape)).reshape(shape)
    return S


def _speeds(S, nod):
    """Largest characteristic speed of the active faces, per axis."""
    h = S["h"].clamp_min(DRY)
    u, v, sq = S["hu"] / h, S["hv"] / h, torch.sqrt(h)
    out = []
    for axis in (1, 0):
        n, t = (u, v) if axis else (-v, u)
        (hi, hj), (ui, uj), (vi, vj), (si, sj) = (_sides(q, axis) for q in (h, n, t, sq))
        ut = (ui * si + uj * sj) / (si + sj)
        ct = torch.sqrt(G_ACC * 0.5 * (hi + hj))
        a = 0.5 * sum(_sides(S["G"], axis)) * (ui * ui + ui * uj + uj * uj + vi * vj) / (si * sj)
        coupled = ~(a < 1e-5)
        a1 = torch.where(coupled, a, torch.full_like(a, 1e-3))
        b, c, d = -2 * ut, (1 + a1) * ct * ct - ut * ut, -ct * ct * a1 * ut
        p = -c - b * b / 3
        q = -(2 * b**3 + 9 * b * c + 27 * d) / 27
        x = 1.5 * q / p * torch.sqrt(-3 / p)
        inside = x.abs() < 1
        ang = torch.where(inside, torch.arccos(torch.where(inside, x, torch.zeros_like(x))),
                          torch.where(x > 0, torch.zeros_like(x), torch.full_like(x, math.pi)))
        amp = 2 * torch.sqrt(-p / 3)
        lo = torch.where(coupled, amp * torch.cos((ang + 2 * math.pi) / 3) + b / 3, ut - ct)
        hi_ = torch.where(coupled, amp * torch.cos(ang / 3) + b / 3, ut + ct)
        s = torch.maximum(lo.abs(), hi_.abs())
        s = torch.where(s < VEL, torch.maximum((ut - ct).abs(), (ut + ct).abs()), s)
        (wi, wj), (mi, mj) = _sides(S["h"] > DRY, axis), _sides(nod, axis)
        on = (wi | wj) & ~(mi | mj)
        out.append(torch.where(on, s, torch.zeros_like(s)).reshape(-1))
    return torch.cat(out)


def _exner_init(S, par, nod):
    S = dict(S)
    if par["mpm"]:
        m = par["seds"]
        rough = (m[1] * m[0]).mean() ** (1.0 / 6.0) / 21.1
        S["n_b"] = torch.where(S["z_b"] > SED, rough.expand_as(S["z_b"]), S["n"])
    else:
        S["n_b"] = S["n"]
    S["G"] = _grass(S, par, nod)
    return _handlers(S, par, 0.0)


def _exner_stage(S, dt, par, nod, time):
    h, hu, hv = _exner_hydro(S, dt, par["dx"], nod)
    hu, hv = _corrections(h, hu, hv, S["z"] + S["z_b"], nod)
    S = _handlers(dict(S, h=h, hu=hu, hv=hv), par, time)
    S["G"] = _grass(S, par, nod)
    S["z_b"] = _exner_bed(S, dt, par["dx"], nod)
    return _handlers(S, par, time)


def _mean(a, b):
    return {f: a[f] if a[f] is b[f] else 0.5 * a[f] + 0.5 * b[f] for f in a}


def _exner_dt(S, par, nod):
    return (CFL * par["dx"] / _speeds(S, nod).amax()).clamp_min(1e-6)


def _exner_steps(S, par, nod, scheme, steps):
    dts, time = [], 0.0
    for _ in range(steps):
        dt = _exner_dt(S, par, nod)
        T = _exner_stage(S, dt, par, nod, time)
        S = _mean(S, _exner_stage(T, dt, par, nod, time)) if scheme == "SSPRK2" else T
        dts.append(dt)
    return S, torch.stack(dts)


def _par(bounds, seds, dx):
    nx = bounds.shape[1]
    handlers = []
    for hd in bounds.handlers:
        (by, bx), (iy, ix) = hd["cells"], hd["donors"]
        cells = tuple(torch.from_numpy(np.asarray(y, dtype=np.int64) * nx + np.asarray(x, dtype=np.int64)).cuda()
                      for y, x in ((by, bx), (iy, ix)))
        handlers.append(dict(name=hd["name"], kind=hd["kind"], normal=hd["normal"], values=hd["values"], cells=cells))
    par = dict(handlers=handlers, dx=dx, q={}, mpm=seds is not None)
    if seds is not None:
        par["seds"] = torch.from_numpy(seds).cuda()
    return par


def _nodata(z, bounds):
    m = torch.isnan(z)
    m[0], m[-1], m[:, 0], m[:, -1] = True, True, True, True
    return m & ~torch.from_numpy(bounds.boundary_mask).cuda()


def _rounded(arrs, dtype):
    return {f: v.to(dtype).double() for f, v in arrs.items()}


def _roe_hydro(S, dt, dx):
    """Plain Roe update with the wet / dry thrust and the source limiter."""
    h = torch.where(S["h"] > DRY, S["h"], torch.zeros_like(S["h"]))
    wet = h > 0
    u, v = _div(S["hu"], h, wet), _div(S["hv"], h, wet)
    flux = [0.0, 0.0, 0.0]
    for axis in (1, 0):
        n, t = (u, v) if axis else (-v, u)
        (hi, hj), (ui, uj), (vi, vj), (zi, zj) = (_sides(q, axis) for q in (h, n, t, S["z"]))
        si, sj = torch.sqrt(hi), torch.sqrt(hj)
        half = 0.5 * (hi + hj)
        ht = torch.where(half > DRY, half, torch.zeros_like(half))
        ct = torch.sqrt(G_ACC * ht)
        ut, vt = (ui * si + uj * sj) / (si + sj), (vi * si + vj * sj) / (si + sj)
        lams, ents = [ut - ct, ut, ut + ct], [torch.zeros_like(ut)] * 3
        for k, sign in ((0, -1.0), (2, 1.0)):
            ei, ej = ui + sign * torch.sqrt(G_ACC * hi), uj + sign * torch.sqrt(G_ACC * hj)
            fix = (ei < 0) & (ej > 0)
            for target in ("speed", "entropy"):  # the entropy speed is formed from the replaced one
                val = _div(ei * (ej - lams[k]) if k == 0 else ej * (lams[k] - ei), ej - ei + VEL, fix)
                if target == "speed":
                    lams[k] = torch.where(fix, val, lams[k])
                else:
                    ents[k] = torch.where(fix, lams[k] - val, ents[k])
        l1, l2, l3 = lams
        den = l1 - l3 + VEL
        dh, dq, dr = hj - hi, hj * uj - hi * ui, hj * vj - hi * vi
        a1, a2, a3 = (-l3 * dh + dq) / den, (dr - vt * dh) / ct, (l1 * dh - dq) / den
        dz, di, dj = zj - zi, hi + zi, hj + zj
        step = torch.where((dz >= 0) & (di < zj), hi, torch.where((dz < 0) & (dj < zi), hj, dz))
        full, part = -G_ACC * ht * dz, -G_ACC * (torch.where(dz >= 0, hi, hj) - 0.5 * step.abs()) * step
        thrust = torch.where((dz * (dj - di) >= 0) & (ut * dz > 0), torch.maximum(full, part), part)
        nb = 0.5 * sum(_sides(S["n"], axis))
        slope = nb * nb * torch.sqrt(ut * ut + vt * vt) * ut / (ht ** (4.0 / 3.0)).clamp_min(DRY)
        b1 = (thrust - G_ACC * ht * slope * dx) / den
        b3 = -b1
        h1, h3 = hi + a1 - b1 / l1, hj - a3 + b3 / l3
        m1, m3 = -(hi + a1) * l1.abs(), -(hi - a1) * l3.abs()
        dtf = dx / torch.maximum(torch.maximum(l1.abs(), l2.abs()), l3.abs())
        c1 = (h1 < 0) & (h3 > 0) & (dx / 2 * l1 * (hi / (hi - h1 + VEL)) < dtf)
        b1 = torch.where(c1 & (-m1 >= m3), m1, b1)
        b3 = torch.where(c1, -b1, b3)
        c3 = (h1 > 0) & (h3 < 0) & (dx / 2 * l3 * (hj / (hj - h3 + VEL)) < dtf)
        b3 = torch.where(c3 & (-m3 >= m3), m1, b3)
        b1 = torch.where(c3, -b3, b1)
        P, M = _split(lams, (a1, a2, a3), (b1, 0.0, b3), ents, ct, vt,
                      ((hi < DRY) & (h1 < 0), (hj < DRY) & (h3 < 0)))
        if not axis:
            P, M = (P[0], P[2], -P[1]), (M[0], M[2], -M[1])
        flux = [f + _spread(m, p, axis) for f, m, p in zip(flux, M, P)]
    return [S[f] - dt * q / dx for f, q in zip(("h", "hu", "hv"), flux)]


def _roe_stage(S, dt, par):
    h, hu, hv = _roe_hydro(S, dt, par["dx"])
    return _handlers(dict(S, h=h, hu=hu, hv=hv), par, 0.0)


def _roe_dt(S, dx):
    wet = S["h"] > DRY
    h, hu, hv = (torch.where(wet, S[f], torch.zeros_like(S[f])) for f in ("h", "hu", "hv"))
    c = torch.sqrt(G_ACC * h)
    return CFL * torch.minimum((dx / ((hu / (h + DRY)).abs() + c + VEL)).amin(), (dx / ((hv / (h + DRY)).abs() + c + VEL)).amin())


def _exact_berthon(case, seed):
    x, y, fields, params = _berthon(case, seed)
    X, Y = np.meshgrid(x, y, indexing="xy")
    bounds = BoundaryManager(params, X, Y)
    S = _rounded({f: torch.from_numpy(np.ascontiguousarray(v)).cuda() for f, v in fields.items()}, _dtype(case))
    par, nod = _par(bounds, None, case["dh"]), _nodata(S["z"], bounds)
    S = _exner_init(S, par, nod)
    time, dt, tol, end, freq = 0.0, 0.0, 5e-7, case["end_time"], case["out_freq"]

    def goal(t):
        return min((int(t / freq) + 1) * freq, end)

    while time < end - tol:
        while time + dt < goal(time) - tol:
            d = _exner_dt(S, par, nod)
            S, dt = _exner_stage(S, d, par, nod, time), float(d)
            time += dt
        d = _exner_dt(S, par, nod)
        S, dt = _exner_stage(S, d, par, nod, time), float(d)
        time += dt
    return {f: S[f] for f in FIELDS}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "berthon":
            return _exact_berthon(case, seed)
        if kind == "ensemble":
            ends, dts = [], []
            for (ny, nx), arrs in _members(case, seed):
                bounds = _layout("bed", ny, nx)
                S = _rounded(arrs, _dtype(case))
                par, nod = _par(bounds, _seds(1), DX), _nodata(S["z"], bounds)
                S, d = _exner_steps(_exner_init(S, par, nod), par, nod, case["scheme"], case["steps"])
                ends.append({f: S[f] for f in FIELDS})
                dts.append(d)
            return dict(dts=torch.stack(dts, 1), first=ends[0], last=ends[-1], h=[e["h"] for e in ends[1:-1]],
                        z_b=[e["z_b"] for e in ends[1:-1]])
        S = _rounded(_arrays(case, seed), _dtype(case))
        ny, nx = case["ny"], case["nx"]
        if kind == "roe":
            par = _par(_layout("roe", ny, nx), None, 1.0 / 256)
            dts = []
            for _ in range(case["steps"]):
                dt = _roe_dt(S, par["dx"])
                T = _roe_stage(S, dt, par)
                S = _mean(S, _roe_stage(T, dt, par)) if case["scheme"] == "SSPRK2" else T
                dts.append(dt)
            return dict({f: S[f] for f in ("h", "hu", "hv", "z", "n")}, dts=torch.stack(dts))
        bounds = _layout("ldomain" if kind == "ldomain" else "bed", ny, nx, kind == "vjp" or bool(case.get("inflow")))
        mpm = case.get("grass", "MPM") == "MPM"
        par, nod = _par(bounds, _seds(case.get("nsed", 1)) if mpm else None, DX), _nodata(S["z"], bounds)
        if kind in ("bed", "ldomain"):
            S, dts = _exner_steps(_exner_init(S, par, nod), par, nod, case["scheme"], case["steps"])
            return dict({f: S[f] for f in FIELDS}, dts=dts)
    if kind == "jvp":
        dot = _direction(case, seed)
        with fwAD.dual_level(), torch.no_grad():
            S = {f: fwAD.make_dual(v, dot.get(f, torch.zeros_like(v))) for f, v in S.items()}
            S, dts = _exner_steps(_exner_init(S, par, nod), par, nod, case["scheme"], case["steps"])
            both = {f: fwAD.unpack_dual(S[f]) for f in FIELDS}
            d = fwAD.unpack_dual(dts)
            zero = torch.zeros_like(both["h"].primal)
            return dict(value={f: both[f].primal for f in FIELDS}, dts=d.primal, dts_dot=d.tangent,
                        dot={f: both[f].tangent if both[f].tangent is not None else zero for f in ("h", "hu", "hv", "z_b", "G")})
    if case["ny"] * case["nx"] * case["steps"] > 300_000 * 16:
        return None
    leaves = {f: S[f].requires_grad_() for f in ("h", "hu", "hv", "z_b")}
    d50 = par["seds"][1].clone().requires_grad_()
    q = torch.tensor(0.3, dtype=torch.float64, device="cuda", requires_grad=True)
    par["seds"] = torch.cat([par["seds"][:1], d50[None], par["seds"][2:]])
    par["q"] = {hd["name"]: q for hd in par["handlers"] if hd["kind"].endswith("ConstantInflux")}
    with torch.enable_grad():
        S, _ = _exner_steps(_exner_init(dict(S, **leaves), par, nod), par, nod, case["scheme"], case["steps"])
        cost = ((S["z"] + S["z_b"] - _target(case, seed)) ** 2).sum()
        g = torch.autograd.grad(cost, [leaves[f] for f in ("h", "hu", "hv", "z_b")] + [d50, q])
    return dict(cost=cost.detach(), grad=dict(zip(("h", "hu", "hv", "z_b"), g[:4])), d50=g[4], inflow=float(g[5]))
