"""The workloads this package is measured on, through its public entry points.

Kinds of case and the program each stands for:

* ``solve``  -- ``fdtd.FDTD``: material arrays on the host, ``solve_forward``,
  then the raw phasors of the whole grid.  Fixed step counts (the time loop as
  such) or a run to the tolerance (``steps`` = 0).
* ``monitor`` -- the same with ``field_domains``: a program that reads the
  interpolated fields on its monitor planes and the source power.
* ``handle`` -- ``serving.Request`` and ``FDTD_solve_cw``: permittivity built on
  the GPU, phasors left in device memory.
* ``serve``  -- ``serving.run_stream``: requests of mixed grids and wavelengths
  through one ``ServeEngine``.
* ``gradient`` -- ``adjoint.mmi_objective``: figure of merit and its gradient by
  a forward and an adjoint solve.
* ``mode``   -- ``modes.ModeFullVector``: modes of a waveguide cross-section and
  the current source that launches one.
* ``layers`` -- ``grid.StructuredMaterial3D.get_values`` at the Yee positions:
  what building a simulation of layered, patterned materials costs.

``exact`` steps the same Yee grid in plain float64 torch.
"""
import ctypes
import math

import numpy as np
import torch

EPS_SI, EPS_SIO2 = 12.25, 2.085
YEE = ((0.5, 0.0, -0.5), (0.0, 0.5, -0.5), (0.0, 0.0, 0.0))
DEV = "cuda"


def listed():
    return [
        # the smallest single solve of the serving range: per-step latency and launches
        dict(name="box_64_f32", kind="handle", nx=64, ny=64, nz=64, d=0.04, wavelength=1.55, pml=15,
             precision=32, steps=500, scene="boxes"),
        # the plain float64 solve: a straight strip waveguide, 4000 steps
        dict(name="waveguide_f64", kind="solve", nx=101, ny=76, nz=65, d=0.04, wavelength=1.55, pml=15,
             precision=64, steps=4000, scene="guide", bc="000", lossy=False, mu=False),
        # the headline solve: a 5.2 M-cell planar device in float32, monitors and source power read
        dict(name="device_f32", kind="monitor", nx=321, ny=161, nz=101, d=0.025, wavelength=1.55, pml=20,
             precision=32, steps=1000, scene="device", bc="000", lossy=False, mu=False),
        # the same device in float64
        dict(name="device_f64", kind="handle", nx=321, ny=161, nz=101, d=0.025, wavelength=1.55, pml=20,
             precision=64, steps=400, scene="boxes"),
        # a whole call: the device at half resolution, run to the tolerance
        dict(name="device_half_converging", kind="monitor", nx=161, ny=81, nz=51, d=0.05, wavelength=1.55,
             pml=10, precision=64, steps=0, scene="device", bc="000", lossy=False, mu=False),
        # a wide layered slab with etched trenches, mostly interior: the largest grid
        dict(name="slab_f32", kind="handle", nx=801, ny=401, nz=201, d=0.03, wavelength=1.55, pml=20,
             precision=32, steps=100, scene="slab"),
        # a quarter device behind two symmetry planes, absorbing and magnetic media, odd sizes
        dict(name="quarter_lossy_f64", kind="solve", nx=149, ny=87, nz=59, d=0.03, wavelength=1.31, pml=12,
             precision=64, steps=400, scene="boxes", bc="0EH", lossy=True, mu=True),
        # the same kind of problem in float32
        dict(name="quarter_lossy_f32", kind="solve", nx=203, ny=111, nz=67, d=0.025, wavelength=1.55, pml=13,
             precision=32, steps=400, scene="boxes", bc="0HE", lossy=True, mu=False),
        # continuous batching: eight requests between 64^3 and 384 x 256 x 128 side by side
        dict(name="serve_8", kind="serve", count=8, lo=64, nx=384, ny=256, nz=128, pml=15, steps=64),
        # one optimisation step of a design: forward solve, adjoint solve, overlap
        dict(name="gradient_f32", kind="gradient", d=0.05, pml=10, nd=80, precision=32, steps=600),
        # the mode source of the device's input guide
        dict(name="mode_source", kind="mode", n=161, m=101, d=0.025, neigs=4),
        # the six Yee arrays of a layered, patterned device
        dict(name="layers", kind="layers", nx=321, ny=161, nz=101, d=0.025, prims=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["handle", "handle", "solve", "solve", "monitor", "serve", "gradient", "mode", "layers"])
    d = rng.choice([0.02, 0.025, 0.03, 0.04])
    wl = round(rng.uniform(1.50, 1.60), 3) if rng.random() < 0.7 else 1.31
    if kind in ("handle", "solve", "monitor"):
        big = kind == "handle"
        nx, ny, nz = _log(rng, 56, 800 if big else 330), _log(rng, 48, 400 if big else 170), _log(rng, 44, 200 if big else 110)
        pml = rng.randint(8, 20)
        cells = nx * ny * nz
        steps = max(60, min(1500, int(2.5e9 / cells)))
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz, d=d, wavelength=wl, pml=pml, precision=rng.choice([32, 32, 64]),
                 steps=rng.randint(60, steps), scene="boxes")
        if kind == "handle":
            return dict(c, scene=rng.choice(["boxes", "slab"]))
        lossy = kind == "solve" and rng.random() < 0.5
        return dict(c, scene="device" if kind == "monitor" else rng.choice(["boxes", "guide", "device"]),
                    bc="000" if kind == "monitor" else rng.choice(["000", "0EH", "0H0", "00E", "EH0"]), lossy=lossy,
                    mu=lossy and rng.random() < 0.5)
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(3, 8), lo=64, nx=_log(rng, 80, 384), ny=_log(rng, 80, 256),
                    nz=_log(rng, 70, 128), pml=rng.randint(8, 15), steps=rng.randint(33, 64))
    if kind == "gradient":
        return dict(kind=kind, d=0.05, pml=rng.randint(7, 10), nd=rng.choice([40, 60, 80]),
                    precision=rng.choice([32, 64]), steps=rng.randint(200, 600))
    if kind == "mode":
        return dict(kind=kind, n=rng.randint(61, 161), m=rng.randint(45, 101), d=rng.choice([0.025, 0.03, 0.04]),
                    neigs=rng.choice([1, 2, 4]))
    return dict(kind=kind, nx=_log(rng, 90, 400), ny=_log(rng, 60, 200), nz=_log(rng, 40, 110), d=d,
                prims=rng.randint(6, 32))


# ---------------------------------------------------------------- the scenes
def _extent(case):
    return [(case[k] - 1) * case["d"] for k in ("nx", "ny", "nz")]


def _boxes(case, rng):
    """(x0, x1, y0, y1, z0, z1, eps) in um, painted in order over SiO2."""
    X, Y, Z = _extent(case)
    big = 1e3
    if case["scene"] == "guide":
        yc, zc = Y / 2 + rng.uniform(-0.05, 0.05), Z / 2
        w = rng.uniform(0.45, 0.55)
        return [(-big, big, yc - w / 2, yc + w / 2, zc - 0.11, zc + 0.11, EPS_SI)]
    if case["scene"] == "slab":
        z0 = 0.55 * Z
        out = [(-big, big, -big, big, -big, 0.25 * Z, EPS_SI), (-big, big, -big, big, z0, z0 + 0.22, EPS_SI)]
        for xc in np.sort(rng.uniform(0.25 * X, 0.75 * X, 40)):
            w = rng.uniform(0.1, 0.4)
            out.append((xc - w / 2, xc + w / 2, -big, big, z0 + 0.11, z0 + 0.22 + 1e-9, EPS_SIO2))
        return out
    out = []
    for _ in range(int(rng.integers(3, 13))):
        s, c = rng.uniform(0.2, 2.0, 3), [rng.uniform(0, L) for L in (X, Y, Z)]
        eps = EPS_SI if rng.random() < 0.5 else EPS_SIO2
        out.append((c[0] - s[0] / 2, c[0] + s[0] / 2, c[1] - s[1] / 2, c[1] + s[1] / 2, c[2] - s[2] / 2,
                    c[2] + s[2] / 2, eps))
    return out


def _axes(case, off):
    n = (case["nx"], case["ny"], case["nz"])
    return [(torch.arange(n[a], device=DEV, dtype=torch.float64) + off[a]) * case["d"] for a in range(3)]


def _paint(case, boxes, off, base=EPS_SIO2):
    x, y, z = _axes(case, off)
    e = torch.full((case["nz"], case["ny"], case["nx"]), base, dtype=torch.float64, device=DEV)
    for x0, x1, y0, y1, z0, z1, v in boxes:
        m = ((z >= z0) & (z <= z1))[:, None, None] & ((y >= y0) & (y <= y1))[None, :, None] & \
            ((x >= x0) & (x <= x1))[None, None, :]
        e.masked_fill_(m, v)
    return e


def _device(case, rng, off):
    """A layer with access guides and a design region of a smoothed, projected
    random density."""
    X, Y, Z = _extent(case)
    rho = torch.as_tensor(rng.uniform(0.0, 1.0, (120, 80)))
    k = torch.ones(1, 1, 9, 9, dtype=torch.float64) / 81
    rho = torch.nn.functional.conv2d(rho[None, None], k, padding=4)[0, 0]
    rho = (0.5 + 0.5 * torch.tanh(40.0 * (rho - 0.5))).to(DEV)
    x, y, z = _axes(case, off)
    hx, hy = 0.1875 * X, 0.25 * Y
    inx, iny = (x - X / 2).abs() <= hx, (y - Y / 2).abs() <= hy
    ix = ((x - X / 2 + hx) / (2 * hx) * 120).long().clamp(0, 119)
    iy = ((y - Y / 2 + hy) / (2 * hy) * 80).long().clamp(0, 79)
    guide = ((y - (Y / 2 - 0.125 * Y)).abs() <= 0.25) | ((y - (Y / 2 + 0.125 * Y)).abs() <= 0.25)
    e = EPS_SIO2 + (EPS_SI - EPS_SIO2) * (guide[:, None] & ~inx[None, :]).to(torch.float64)
    e = torch.where(iny[:, None] & inx[None, :], EPS_SIO2 + (EPS_SI - EPS_SIO2) * rho[ix][:, iy].T, e)
    lay = (z - Z / 2).abs() <= 0.11
    return torch.where(lay[:, None, None], e[None], torch.tensor(EPS_SIO2, dtype=torch.float64, device=DEV))


def _materials(case, seed):
    """eps_x, eps_y, eps_z, mu_x, mu_y, mu_z on the GPU, complex128 [Nz][Ny][Nx]."""
    out = []
    for off in YEE:
        rng = np.random.default_rng(seed)
        if case["scene"] == "device":
            e = _device(case, rng, off)
        else:
            e = _paint(case, _boxes(case, rng), off)
        if case.get("lossy"):
            out.append(torch.complex(e, 0.3 * (e > 6.0).to(torch.float64)))
        else:
            out.append(e.to(torch.complex128))
    for off in ((0.0, 0.5, 0.0), (0.5, 0.0, 0.0), (0.5, 0.5, -0.5)):
        if case.get("mu"):
            rng = np.random.default_rng(seed + 1000)
            b = [(*b[:6], float(rng.uniform(1.0, 1.5))) for b in _boxes(case, rng)]
            out.append(_paint(case, b, off, 1.0).to(torch.complex128))
        else:
            out.append(torch.ones((case["nz"], case["ny"], case["nx"]), dtype=torch.complex128, device=DEV))
    return out


def _sheet(case, seed):
    """(x index, Jy profile [Nz][Ny]) of the Gaussian current sheet."""
    X, Y, Z = _extent(case)
    yc = Y / 2 if case["scene"] != "device" else Y / 2 - 0.125 * Y
    w0 = 2.0 if case["scene"] == "slab" else 0.4
    z, y = np.arange(case["nz"]) * case["d"], np.arange(case["ny"]) * case["d"]
    ph = np.random.default_rng(seed + 7).uniform(-0.3, 0.3)
    Zg, Yg = np.meshgrid(z, y, indexing="ij")
    p = np.exp(-((Yg - yc) ** 2 + (Zg - Z / 2) ** 2) / w0 ** 2) * np.exp(1j * ph * Yg)
    return min(case["pml"] + 5, case["nx"] - 2), p


def _length(n, d):
    return (n - 1.5) * d       # ceil(L / d) + 1 = n


# ------------------------------------------------------------------ prepare
def _solver(case, seed):
    from emopt_b200.fdtd import FDTD
    from emopt_b200.misc import DomainCoordinates
    d, n = case["d"], (case["nx"], case["ny"], case["nz"])
    sim = FDTD(_length(n[0], d), _length(n[1], d), _length(n[2], d), d, d, d, case["wavelength"], rtol=1e-6,
               complex_eps=case["lossy"], precision="fp%d" % case["precision"])
    sim.set_pml_cells([case["pml"]] * 6)
    if case["bc"] != "000":
        sim.bc = case["bc"]
    sim.fixed_steps = case["steps"] or None
    mats = [m.cpu().numpy() for m in _materials(case, seed)]
    sim.set_material_arrays(mats[:3], mats[3:])
    k, prof = _sheet(case, seed)
    src = [np.zeros((n[2], n[1], 1), dtype=np.complex128) for _ in range(6)]
    src[1][:, :, 0] = prof
    sim.set_sources(tuple(src), DomainCoordinates.from_indices(k, k + 1, 0, n[1], 0, n[2], d, d, d))
    if case["kind"] == "monitor":
        w = case["pml"]
        D = lambda *a: DomainCoordinates.from_indices(*a, d, d, d)
        ko, zm = n[0] - w - 5, n[2] // 2
        sim.field_domains = [D(ko, ko + 1, w, n[1] - w, w, n[2] - w), D(w, n[0] - w, w, n[1] - w, zm, zm + 1)]
    return sim


def _spec(case, seed, rid=0):
    from emopt_b200.serving import RequestSpec
    rng = np.random.default_rng(seed)
    X, Y, Z = _extent(case)
    k, _ = _sheet(case, seed)
    ph = np.random.default_rng(seed + 7).uniform(-0.3, 0.3)
    return RequestSpec(rid, (case["nz"], case["ny"], case["nx"]), case["d"], case["wavelength"], _boxes(case, rng),
                       w_pml=case["pml"], src_k=k, src_yz=(Y / 2, Z / 2),
                       src_w0=2.0 if case["scene"] == "slab" else 0.4, src_phase_y=ph, fixed_steps=case["steps"],
                       precision=case["precision"])


def _requests(case, seed):
    """The requests of a served batch, as cases of their own."""
    rng = np.random.default_rng(seed * 31 + 5)
    out = []
    for q in range(case["count"]):
        n = [int(round(case["lo"] * (case[k] / case["lo"]) ** min(1.0, 0.12 * ((q + a) % 3) + 0.8 * q / case["count"])))
             for a, k in enumerate(("nx", "ny", "nz"))]
        out.append(dict(kind="handle", nx=n[0], ny=n[1], nz=n[2], d=(0.04, 0.025, 0.02)[q % 3],
                        wavelength=float(rng.uniform(1.50, 1.60)), pml=case["pml"], precision=32,
                        steps=case["steps"], scene="boxes"))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "monitor"):
        return dict(kind=kind, sim=_solver(case, seed))
    if kind == "handle":
        from emopt_b200 import serving
        spec = _spec(case, seed)
        ones = torch.ones(spec.ncells, dtype=torch.complex128, device=DEV)
        req = serving.Request(spec, 0, ones)
        req.set_outputs()
        return dict(kind=kind, req=req, ones=ones)
    if kind == "serve":
        from emopt_b200 import serving
        specs = [_spec(c, seed + 17 * q, q) for q, c in enumerate(_requests(case, seed))]
        return dict(kind=kind, specs=specs, engine=serving.ServeEngine(0, 60e9, 16, 32))
    if kind == "gradient":
        from emopt_b200 import adjoint, problems
        p = problems.mmi_gradient(seed=seed, nd=(case["nd"],) * 2, d=case["d"], w_pml=case["pml"],
                                  fixed_steps=case["steps"])
        obj, params = adjoint.mmi_objective(p, "fp%d" % case["precision"])
        return dict(kind=kind, obj=obj, params=params)
    if kind == "mode":
        from emopt_b200 import grid
        from emopt_b200.misc import DomainCoordinates
        rng, d = np.random.default_rng(seed), case["d"]
        n, m = case["n"], case["m"]
        Xs, Ys, Zs = 60 * d, (n - 1) * d, (m - 1) * d
        yc, w = Ys / 2 + rng.uniform(0.1, 0.3), rng.uniform(0.45, 0.6)
        prims = [(grid.Rectangle(Xs / 2, yc, 2 * Xs, w), EPS_SI, Zs / 2 - 0.13, Zs / 2 + 0.09, 1),
                 (grid.Rectangle(Xs / 2, Ys / 2, 2 * Xs, 2 * Ys), EPS_SIO2, -Zs, Zs / 2 + 0.2, 2),
                 (grid.Rectangle(Xs / 2, Ys / 2, 2 * Xs, 2 * Ys), 1.0, Zs / 2 + 0.2, 2 * Zs, 3)]
        eps = grid.StructuredMaterial3D(Xs, Ys, Zs, d, d, d)
        for p, v, z1, z2, layer in prims:
            p.layer, p.material_value = layer, v
        for p, v, z1, z2, layer in reversed(prims):
            eps.add_primitive(p, z1, z2)
        return dict(kind=kind, eps=eps, mu=grid.ConstantMaterial3D(1.0), neigs=case["neigs"], d=d,
                    plane=DomainCoordinates.from_indices(30, 31, 0, n, 0, m, d, d, d))
    from emopt_b200 import grid
    rng, d = np.random.default_rng(seed), case["d"]
    X, Y, Z = _extent(case)
    mat = grid.StructuredMaterial3D(X, Y, Z, d, d, d)
    back = grid.Rectangle(X / 2, Y / 2, 4 * X, 4 * Y)
    back.layer, back.material_value = 1000, EPS_SIO2
    mat.add_primitive(back, -Z, 2 * Z)
    bus = grid.Rectangle(X / 2, Y / 2 + rng.uniform(-0.1, 0.1), 4 * X, 0.5)
    bus.layer, bus.material_value = 999, EPS_SI
    mat.add_primitive(bus, Z / 2 - 0.11, Z / 2 + 0.11)
    cols = (case["prims"] + 2) // 3
    for q in range(case["prims"]):                    # a pattern of rectangles, tapers and scatterers
        x, y = X * (q // 3 + rng.uniform(0.45, 0.55)) / cols, Y * (q % 3 + rng.uniform(0.45, 0.55)) / 3
        s = rng.uniform(0.2, 0.4) * min(X / cols, Y / 3)
        if q % 4 == 0:
            p = grid.Rectangle(x, y, 1.6 * s, rng.uniform(0.6, 1.8) * s)
        elif q % 4 == 1:
            p = grid.Polygon(x + s * np.array([-1.0, 1.0, 1.0, -1.0]), y + s * np.array([-0.3, -0.9, 0.9, 0.3]))
        else:
            t = 2 * np.pi * (np.arange(5 + q % 4) + rng.uniform(0, 1)) / (5 + q % 4)
            p = grid.Polygon(x + s * np.cos(t), y + s * np.sin(t))
        p.layer, p.material_value = q + 1, EPS_SI if q % 4 else 4.0
        mat.add_primitive(p, Z / 2 - 0.11, Z / 2 + (0.11 if q % 2 else 0.0))
    return dict(kind="layers", mat=mat, n=(case["nx"], case["ny"], case["nz"]))


# ---------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind in ("solve", "monitor"):
        sim = state["sim"]
        sim.solve_forward()
        if kind == "solve":
            return [sim.get_field(c) for c in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")]
        return dict(fields=[list(f) for f in sim.saved_fields], power=sim.source_power)
    if kind == "handle":
        from emopt_b200 import fdtd_ctypes as ct
        req, res = state["req"], ct.SolveResult()
        if ct.libFDTD.FDTD_solve_cw(req.h, ctypes.byref(req.opt), ctypes.byref(res)) not in (ct.FDTD_OK, ct.FDTD_NMAX):
            raise RuntimeError(ct.last_error(req.h)[1])
        return req.out
    if kind == "serve":
        from emopt_b200 import serving
        got = {}
        serving.run_stream(state["specs"], state["engine"], realtime=False,
                           on_done=lambda req, r: got.__setitem__(req.spec.rid, list(req.out)))
        return [got[s.rid] for s in state["specs"]]
    if kind == "gradient":
        x = state["params"].clone().requires_grad_(True)
        f = state["obj"](x)
        f.backward()
        return dict(fom=f.detach(), grad=x.grad)
    if kind == "mode":
        from emopt_b200.modes import ModeFullVector
        m = ModeFullVector(1.55, state["eps"], state["mu"], state["plane"], n0=3.0, neigs=state["neigs"], verbose=False)
        m.build()
        m.solve()
        d = state["d"]
        return dict(neff=np.array(m.neff), source=list(m.get_source(0, d, d, d)))
    K, J, I = state["n"]
    return [state["mat"].get_values(0, K, 0, J, 0, I, sx=o[0], sy=o[1], sz=o[2], device=0) for o in YEE]


# --------------------------------------------------------------------- work
def _timing(case):
    nl = case["wavelength"] / case["d"]
    return nl, nl * math.sqrt(3.0), int(nl * math.sqrt(3.0) * 3 / 4)


def _step_bytes(nx, ny, nz, pml, size, lossy=False, mu=False):
    """One time step: six fields read and written, three E coefficients read
    (six when lossy, three more for a varying mu), four CPML accumulators per
    slab that holds the cell read and written."""
    cells = nx * ny * nz
    slab = 2 * pml * (ny * nz + nx * nz + nx * ny)
    return size * (cells * (15 + 3 * lossy + 3 * mu) + 8 * slab)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "monitor", "handle"):
        steps = case["steps"] or 4200
        n = steps + 2 * _timing(case)[2]
        cells = case["nx"] * case["ny"] * case["nz"]
        b = _step_bytes(case["nx"], case["ny"], case["nz"], case["pml"], case["precision"] // 8,
                        bool(case.get("lossy")), bool(case.get("mu")))
        return {"bytes": n * b + cells * 16 * 12, "flops": n * cells * 40}
    if kind == "serve":
        w = [work(c) for c in _requests(case, 1)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if kind == "gradient":
        n = [int(math.ceil(L / case["d"]) + 1) for L in (8.0, 4.0, 2.5)]
        c = dict(kind="handle", nx=n[0], ny=n[1], nz=n[2], pml=case["pml"], precision=case["precision"],
                 steps=case["steps"], wavelength=1.55, d=case["d"])
        w = work(c)
        return {"bytes": 2 * w["bytes"], "flops": 2 * w["flops"]}
    if kind == "mode":
        # inverses of the line blocks (6 L unknowns each), and one reading of
        # them per application of the operator, about 40 applications per mode
        L, lines = min(case["n"], case["m"]), max(case["n"], case["m"])
        nb = 6 * L
        return {"bytes": 40 * case["neigs"] * lines * nb * nb * 16, "flops": 8 * lines * nb ** 3}
    return {"bytes": 3 * 16 * case["nx"] * case["ny"] * case["nz"],
            "flops": 3 * 100 * case["nx"] * case["ny"] * case["nz"]}


# -------------------------------------------------------------------- exact
def _ramp(n, pml, axis, dt, half):
    """CPML (b, c) along one axis (sigma 3, alpha 0, kappa 1, cubic ramp) for the
    H or the E update, zero outside the slabs: psi <- b psi + c d."""
    b, c = torch.ones(n, dtype=torch.float64), torch.zeros(n, dtype=torch.float64)
    edge = n - pml
    for k in range(n):
        if k < pml:
            q = pml - 1 - k
            dist = (q - 0.5 if half == "H" else q) if axis != 2 else (q if half == "H" else q + 0.5)
        elif (k >= edge) if axis != 2 else (k > edge):
            q = k - edge
            dist = (q + 0.5 if half == "H" else q) if axis != 2 else (q if half == "H" else q - 0.5)
        else:
            continue
        f = max(0.0, dist / pml) ** 3
        b[k] = math.exp(-dt * 3.0 * f)
        c[k] = 0.0 if b[k] == 1.0 else b[k] - 1.0
    return b.to(DEV), c.to(DEV)


def _fields(case, seed):
    """The complex steady-state fields of a fixed-length solve, float64 torch."""
    nx, ny, nz, d, w, bc = case["nx"], case["ny"], case["nz"], case["d"], case["pml"], case.get("bc", "000")
    R = case["wavelength"] / (2 * math.pi)
    dt = 0.95 * d / R / math.sqrt(3.0)
    ncycle = case["wavelength"] / d * math.sqrt(3.0)
    Tn, T, m = int(np.int64(ncycle * 3 / 4)), ncycle * 20.0 * dt, 1e-4
    kk = T * T / math.log((1 + m) / m)
    o = R / d
    mats = _materials(case, seed)
    a = b = None
    if case.get("lossy"):
        den = [e.real / dt + e.imag / 2 for e in mats[:3]]
        a = [(e.real / dt - e.imag / 2) / q for e, q in zip(mats[:3], den)]
        b = [1.0 / q for q in den]
    else:
        b = [dt / e.real for e in mats[:3]]
    bh = [dt / q.real if case.get("mu") else dt for q in mats[3:]]
    del mats
    k_src, prof = _sheet(case, seed)
    amp, ph = torch.as_tensor(np.abs(prof), device=DEV), torch.as_tensor(-np.angle(prof), device=DEV)
    ar, ai = amp * torch.cos(ph) * b[1][:, :, k_src], amp * torch.sin(ph) * b[1][:, :, k_src]
    shape = (nz, ny, nx)
    E = [torch.zeros(shape, dtype=torch.float64, device=DEV) for _ in range(3)]
    H = [torch.zeros(shape, dtype=torch.float64, device=DEV) for _ in range(3)]
    D = torch.empty(shape, dtype=torch.float64, device=DEV)
    N, DIM = (nx, ny, nz), (2, 1, 0)          # axis -> tensor dimension
    tab = {h: [_ramp(N[x], w, x, dt, h) for x in range(3)] for h in "HE"}

    def cut(t, x, s):
        return t[(slice(None),) * DIM[x] + (s,)]

    def slabs(x):
        return [slice(0, w), slice(N[x] - w + (1 if x == 2 else 0), N[x])]

    def view(t, x):
        return t.view([-1 if q == DIM[x] else 1 for q in range(3)])

    psi = {h: {} for h in "HE"}

    def add(dst, F, x, half, sign, coef):
        """dst += sign coef (dF/dx + CPML correction); forward differences for
        the H update, backward ones for the E update."""
        lo, hi = slice(0, N[x] - 1), slice(1, N[x])
        if half == "H":
            torch.sub(cut(F, x, hi), cut(F, x, lo), out=cut(D, x, lo))
            torch.neg(cut(F, x, slice(N[x] - 1, N[x])), out=cut(D, x, slice(N[x] - 1, N[x])))
        else:
            torch.sub(cut(F, x, hi), cut(F, x, lo), out=cut(D, x, hi))
            first, ghost = cut(F, x, slice(0, 1)), {"0": 1.0, "E": 2.0, "H": 0.0}[bc[x]]
            torch.mul(first, ghost, out=cut(D, x, slice(0, 1)))
        D.mul_(o)
        tb, tc = tab[half][x]
        for s in slabs(x):
            key = (x, id(dst), s.start)
            g = cut(D, x, s)
            p = psi[half].get(key)
            if p is None:
                p = psi[half][key] = torch.zeros_like(g)
            p.mul_(view(tb[s], x)).add_(view(tc[s], x) * g)
            g.add_(p)
        if isinstance(coef, float):
            dst.add_(D, alpha=sign * coef)
        else:
            dst.addcmul_(D, coef, value=sign)

    snaps = []
    total = case["steps"] + 2 * Tn
    for n in range(total):
        add(H[0], E[1], 2, "H", 1.0, bh[0]); add(H[0], E[2], 1, "H", -1.0, bh[0])
        add(H[1], E[2], 0, "H", 1.0, bh[1]); add(H[1], E[0], 2, "H", -1.0, bh[1])
        add(H[2], E[0], 1, "H", 1.0, bh[2]); add(H[2], E[1], 0, "H", -1.0, bh[2])
        if a is not None:
            for c in range(3):
                E[c].mul_(a[c])
        add(E[0], H[2], 1, "E", 1.0, b[0]); add(E[0], H[1], 2, "E", -1.0, b[0])
        add(E[1], H[0], 2, "E", 1.0, b[1]); add(E[1], H[2], 0, "E", -1.0, b[1])
        add(E[2], H[1], 0, "E", 1.0, b[2]); add(E[2], H[0], 1, "E", -1.0, b[2])
        t = (n + 0.5) * dt
        env = (1 + m) * math.exp(-(t - T) ** 2 / kk) - m if t <= T else 1.0
        E[1][:, :, k_src] -= env * (math.sin(t) * ar + math.cos(t) * ai)
        if n + 1 in (case["steps"], case["steps"] + Tn):
            snaps.append([f.clone() for f in E + H])
    snaps.append(E + H)
    out = []
    for c in range(6):
        ts = [(case["steps"] + q * Tn) * dt - (0.5 * dt if c >= 3 else 0.0) for q in range(3)]
        s, co = [math.sin(t) for t in ts], [math.cos(t) for t in ts]
        f10, f21 = snaps[1][c] - snaps[0][c], snaps[2][c] - snaps[1][c]
        Yv = f10 * (s[2] - s[1]) - f21 * (s[1] - s[0])
        Xv = f21 * (co[1] - co[0]) - f10 * (co[2] - co[1])
        late = f21 * f21 >= f10 * f10
        f = torch.where(late, f21, f10)
        late = late.to(torch.float64)
        ds = late * (s[2] - s[1]) + (1.0 - late) * (s[1] - s[0])
        dc = late * (co[2] - co[1]) + (1.0 - late) * (co[1] - co[0])
        g = f / (Xv * ds + Yv * dc)
        ok = (f10 != 0) | (f21 != 0)
        out.append(torch.complex(torch.where(ok, g * Xv, 0.0), torch.where(ok, -g * Yv, 0.0)))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "handle"):
        F = _fields(case, seed)
        return [f.cpu().numpy() for f in F] if kind == "solve" else F
    if kind == "serve":
        # about 250 small steps per request: a few seconds in all
        return [_fields(c, seed + 17 * q) for q, c in enumerate(_requests(case, seed))]
    return None
