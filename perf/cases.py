"""Workloads that stand for what the engine is used for, at sizes from a few thousand cells to 10^8.

Every case is driven through the public Python API (Simulation and
batch_forward_adjoint).  A state is a run in progress: smooth wave packets in
the interior of the grid, a pulse on its way from the source, the monitors a
user would set.  run() advances the state and reads what such a program reads,
so a second run() continues where the first one stopped.  exact() states the
same update equations in plain torch at 64 bits.
"""
import math

import numpy as np
import torch

from dtmaxwell4_b200 import Simulation, abi
from dtmaxwell4_b200.engine import batch_forward_adjoint

EX, EY, EZ, HX, HY, HZ = range(6)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a design sketch or a unit check of a user's script: one small box, the launches are all there is
        dict(name="dipole_48", kind="dipole", nx=48, ny=48, nz=48, steps=100, pml=8, order=2, engine="default"),
        # the 128^3 point-dipole configuration: dielectric sphere, 10-cell CPML, Ez/Hx traces at 8 points
        dict(name="dipole_128", kind="dipole", nx=128, ny=128, nz=128, steps=200, pml=10, order=2, engine="default"),
        # closed metal cavity of odd extents, no absorber
        dict(name="cavity_odd", kind="cavity", nx=77, ny=201, nz=55, steps=150, pml=0, order=2, engine="default"),
        # two-pole (Lorentz + Drude) ellipsoid on a ragged grid, absorbers of uneven depth, one face without
        dict(name="lorentz_odd", kind="lorentz", nx=149, ny=93, nz=211, steps=96, pml=9, order=2, engine="default"),
        # the 384^3 Drude nanoparticle in a plane-wave TF/SF box with its 16-frequency monitor plane
        dict(name="drude_tfsf_384", kind="drude_tfsf", nx=384, ny=384, nz=384, steps=200, pml=12, order=2, engine="tuned"),
        # a production-size dielectric run
        dict(name="dielectric_large", kind="dipole", nx=640, ny=512, nz=384, steps=32, pml=10, order=2, engine="tuned"),
        # photonic-crystal slab on a gyrotropic layer, 6-face power flux box with 32 frequencies
        dict(name="gyro_flux", kind="gyro", nx=256, ny=256, nz=384, steps=64, pml=10, order=2, engine="tuned"),
        # the fourth-order stencil in a box: Drude particle, plane-wave TF/SF
        dict(name="order4_drude", kind="drude_tfsf", nx=192, ny=160, nz=224, steps=64, pml=10, order=4, engine="default"),
        # the reference's own set-up: its geometry, split PML, fourth order, TF/SF dipole, averaging sensors
        dict(name="reference_mode", kind="reference", nx=180, ny=180, nz=128, steps=66, pml=15, order=4, engine="default"),
        # gradient of a flux objective: design history recorded in the forward pass
        dict(name="gradient", kind="gradient", nx=192, ny=160, nz=128, steps=100, pml=10, order=2, engine="sweep",
             design=48, drude=False, history=True, count=1),
        # gradient next to a metal particle on a ragged grid, checkpoint every 25 steps and recompute
        dict(name="gradient_checkpointed", kind="gradient", nx=171, ny=99, nz=133, steps=100, pml=8, order=2, engine="default",
             design=24, drude=True, history=False, count=1),
        # a batch of gradients of uneven instances
        dict(name="gradient_batch", kind="gradient", nx=128, ny=96, nz=96, steps=60, pml=10, order=2, engine="sweep",
             design=16, drude=False, history=True, count=6),
    ]


def draw(rng):
    def size(lo, hi, most):
        while True:
            n = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
            if n[0] * n[1] * n[2] <= most:
                return n
    kind = rng.choice(("dipole", "dipole", "cavity", "lorentz", "drude_tfsf", "drude_tfsf", "gyro", "reference", "gradient", "gradient"))
    order = 2
    engine = rng.choice(("default", "tuned", "sweep"))
    extra = {}
    if kind == "dipole":
        pml = rng.randint(5, 14)
        n = size(2 * pml + 16, 512, 6e7)
        order = rng.choice((2, 2, 4))
    elif kind == "cavity":
        pml = 0
        n = size(32, 320, 2e7)
        order = rng.choice((2, 2, 4))
    elif kind == "lorentz":
        pml = rng.randint(5, 12)
        n = size(2 * pml + 30, 320, 1.5e7)
    elif kind == "drude_tfsf":
        pml = rng.randint(6, 12)
        n = size(2 * pml + 48, 384, 4e7)
        order = rng.choice((2, 2, 4))
    elif kind == "gyro":
        pml = rng.randint(6, 10)
        n = size(2 * pml + 60, 320, 2e7)
    elif kind == "reference":
        pml, order = 15, 4
        n = size(72, 288, 8e6)
        n[0], n[1] = n[0] // 3 * 3, n[1] // 3 * 3
    else:
        pml = rng.randint(6, 10)
        n = size(2 * pml + 40, 224, 4e6)
        extra = dict(design=rng.randint(8, 20), drude=rng.random() < 0.4, history=rng.random() < 0.6, count=rng.choice((1, 1, 3, 5)))
        order = rng.choice((2, 2, 2, 4))
    if kind == "reference" or order == 4:
        engine = rng.choice(("default", "tuned")) if kind != "gradient" else "default"
    cells = n[0] * n[1] * n[2] * extra.get("count", 1)
    most = 150 if kind != "gradient" else 80
    steps = max(24, min(most, int(2e9 / cells)))
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], steps=steps, pml=pml, order=order, engine=engine, **extra)


# ------------------------------------------------------------------ the set-up of a case, in plain numbers
def _pulse(lambda0):
    f0 = 1.0 / lambda0
    tau = 3.0 * lambda0 / (2.0 * math.sqrt(math.log(2.0)))
    return f0, tau


def _nodes(n, comp, ds=1.0):
    """Node coordinates of E component comp along the three axes (cells)."""
    return [(torch.arange(m, dtype=torch.float64, device="cuda") + (0.0 if a == comp else 0.5)) * ds for a, m in enumerate(n)]


def _ellipsoid(n, comp, centre, radii):
    x = _nodes(n, comp)
    return sum(((x[a] - centre[a]) / radii[a]).square().reshape([-1 if b == a else 1 for b in range(3)]) for a in range(3)) <= 1.0


def _setup(case, seed, which=0):
    """Everything about a case but the initial fields: numbers and material indices."""
    n = (case["nx"], case["ny"], case["nz"])
    kind, pml, order, steps = case["kind"], case["pml"], case["order"], case["steps"]
    rng = np.random.default_rng([seed, which])
    if which:                                         # the further instances of a batch: uneven sizes
        n = tuple(int(m + rng.integers(-m // 6, m // 6 + 1)) for m in n)
    s = dict(n=n, ds=1.0, dt=0.5 if order == 2 else 0.4, order=order, kind=kind, steps=steps, pml=((pml, pml),) * 3, geometry="box",
             absorber="cpml" if pml else "none", materials=[dict(eps=1.0)], idx=None, sources=[], tfsf=None, probes=[], dft=[],
             flux=[], design=None, every=1)
    mid = [m // 2 for m in n]
    small = min(n)
    lambda0 = 20.0
    f0, tau = _pulse(lambda0)
    phase = float(rng.uniform(0.0, 10.0))             # how far the pulse has come
    dipole = dict(comp=EZ, i=mid[0], j=mid[1], k=mid[2], amp=1.0, f0=f0, tau=tau, t0=0.5 * tau + phase)
    inner = [(pml + 1, m - pml - 2) for m in n]

    def points(count):
        return [[int(rng.integers(lo, hi + 1)) for lo, hi in inner] for _ in range(count)]
    if kind in ("dipole", "cavity"):
        s["sources"] = [dipole]
        s["probes"] = [(c, *p, 0) for p in points(8) for c in (EZ, HX)]
        s["materials"].append(dict(eps=4.0))
        s["idx"] = [_ellipsoid(n, c, [0.5 * m for m in n], [0.156 * small] * 3) for c in range(3)]
    elif kind == "lorentz":
        # no absorber below y, uneven depths elsewhere
        s["pml"] = ((pml, max(4, pml - 2)), (0, pml + 2), (pml - 1, pml - 1))
        s["sources"] = [dict(dipole, comp=EX, i=pml + 6, k=mid[2] + 3)]
        s["probes"] = [(c, *p, 0) for p in points(4) for c in range(6)]
        s["materials"] += [dict(eps_inf=2.0, sigma=0.01, poles=[(0, 0.8, 2 * math.pi / 14, 0.02, 0.0), (1, 1.0, 2 * math.pi / 10, 0.03, 0.0)]),
                           dict(eps=(2.25, 2.5, 3.0))]
        ell = [_ellipsoid(n, c, [0.5 * m for m in n], [0.2 * m for m in n]) for c in range(3)]
        s["idx"] = [e.to(torch.uint8) for e in ell]
        for e in s["idx"]:                            # an anisotropic substrate under the ellipsoid, through the absorber
            sub = e[:, :, : n[2] // 5]
            sub[sub == 0] = 2
        s["dft"] = [(1, n[1] // 2 + 3, (EX, EZ, HX), [2 * math.pi * f0 * q for q in (0.8, 1.0, 1.2)])]
    elif kind == "drude_tfsf":
        inset = 20 if small >= 300 else max(6, small // 16)
        wp = 2 * math.pi / 8.0
        s["materials"].append(dict(eps_inf=1.0, sigma=0.0, poles=[(1, 1.0, wp, wp / 100.0, 0.0)]))
        s["idx"] = [_ellipsoid(n, c, [0.5 * m for m in n], [0.104 * small] * 3) for c in range(3)]
        s["tfsf"] = dict(kind="plane", lo=[float(pml + inset)] * 3, hi=[float(m - pml - inset) for m in n], amp=1.0, f0=f0, tau=tau,
                         t0=0.5 * tau + phase)
        df = math.sqrt(math.log(10.0)) / (math.pi * tau)
        s["dft"] = [(0, n[0] - pml - inset // 2, (EY, EZ, HY, HZ), list(2 * math.pi * np.linspace(f0 - df, f0 + df, 16)))]
        s["probes"] = [(EZ, mid[0] + int(0.104 * small) + 4, mid[1], mid[2], 0), (EZ, pml + inset // 2, mid[1], mid[2], 0),
                       (HY, pml + inset + 3, mid[1], mid[2], 0)]
    elif kind == "gyro":
        lam = 32.0 / 0.3
        w0 = 2 * math.pi / lam
        wc = 0.5 * w0
        wp2 = 0.3 * w0 * (w0 * w0 - wc * wc) / wc     # off-diagonal 0.3, diagonal 4 at w0
        s["materials"] += [dict(eps=12.0), dict(eps_inf=4.0 + wp2 / (w0 * w0 - wc * wc), gyro=(math.sqrt(wp2), 0.0, wc)), dict(eps=4.0)]
        slab = max(6, n[2] // 12)
        z0 = mid[2] - slab // 2
        layer = max(8, n[2] // 5)
        s["idx"] = []
        for c in range(3):
            x, y, z = _nodes(n, c)
            a = torch.zeros(n, dtype=torch.uint8, device="cuda")
            # triangular lattice of holes, the one at the dipole left out
            h = 32.0 * math.sqrt(3.0) / 2.0
            hole = torch.zeros(n[:2], dtype=torch.bool, device="cuda")
            for r in range(-n[1] // 27 - 2, n[1] // 27 + 3):
                cy = mid[1] + 0.5 + r * h
                px = (x - (mid[0] + 0.5 + 16.0 * r) + 16.0) % 32.0 - 16.0
                near = px.square()[:, None] + (y - cy).square()[None, :] <= 100.0
                if r == 0:
                    near &= ((x - mid[0] - 0.5).abs() > 16.0)[:, None]
                hole |= near
            zi = torch.nonzero((z >= z0) & (z < z0 + slab)).flatten()
            a[:, :, zi] = torch.where(hole, 0, 1).to(torch.uint8)[:, :, None].expand(n[0], n[1], len(zi))
            zl = torch.nonzero((z >= z0 - layer) & (z < z0)).flatten()
            a[:, :, zl] = 3                           # inside the absorber the layer is a plain dielectric
            k0, k1 = max(int(zl[0]), pml), min(int(zl[-1]) + 1, n[2] - pml)
            a[pml:n[0] - pml, pml:n[1] - pml, k0:k1] = 2
            s["idx"].append(a)
        f0, tau = _pulse(lam)
        s["sources"] = [dict(dipole, f0=f0, tau=tau, t0=0.3 * tau + phase)]
        df = math.sqrt(math.log(10.0)) / (math.pi * tau)
        half = min(20, small // 2 - pml - 4)
        s["flux"] = [([m - half for m in mid], [m + half for m in mid], list(2 * math.pi * np.linspace(f0 - df, f0 + df, 32)))]
        s["probes"] = [(EZ, mid[0] + 3, mid[1] - 2, mid[2], 0)]
    elif kind == "reference":
        ds = 0.005
        s.update(ds=ds, dt=0.002, geometry="reference", absorber="split", pml=((15, 15), (15, 15), (0, 16)), vmax=1 / 1.75, every=22)
        s["materials"] = [dict(eps=1.75 ** 2), dict(eps_inf=1.0, sigma=0.0, poles=[(1, 1.0, 136.66 / 3.0, 2.69e13 / 2 / 3e14, 0.0)]),
                          dict(eps=1.8 ** 2)]
        a = torch.zeros(n, dtype=torch.uint8, device="cuda")
        a[:, :, :8] = 1                               # metal film, thin oxide, organic above
        a[:, :, 8:11] = 2
        s["idx"] = [a, a, a]
        c = 1.0 / 1.75
        half = [5.25 * ds, 5.25 * ds, 4.25 * ds]
        ctr = [n[0] // 2 * ds, n[1] // 2 * ds, 24 * ds]
        s["tfsf"] = dict(kind="dipole", lo=[ctr[q] - half[q] for q in range(3)], hi=[ctr[q] + half[q] for q in range(3)], c=c,
                         w=2 * math.pi * c / (0.2 * float(rng.uniform(0.9, 1.1))), kenv=0.3)
        s["probes"] = [(c, mid[0] + 3 * x, mid[1], 24, 1) for x in range(4) for c in range(6)]
    elif kind == "gradient":
        d = [min(case["design"], m - 2 * pml - 24) for m in n]
        d[2] = max(4, d[2] // 2)
        lo = [(m - q) // 2 for m, q in zip(n, d)]
        s["design"] = (lo, rng.uniform(1.0, 12.0, size=(3, *d)).astype(np.float32))
        s["plane_x"], s["omega"] = n[0] - pml - 4, 2 * math.pi / 24.0
        s["sources"] = [dict(dipole, i=(pml + lo[0]) // 2)]
        s["idx"] = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(3)]
        for b in range(4):                            # dielectric blocks around the design region
            s["materials"].append(dict(eps=float(rng.uniform(1.0, 12.0))))
            at = [int(rng.integers(pml + 1, m - pml - 9)) for m in n]
            for c in range(3):
                s["idx"][c][at[0]:at[0] + 8, at[1]:at[1] + 6, at[2]:at[2] + 7] = len(s["materials"]) - 1
        if case["drude"]:
            wp = 2 * math.pi / 8.0
            s["materials"].append(dict(eps_inf=1.0, sigma=0.0, poles=[(1, 1.0, wp, wp / 100.0, 0.0)]))
            at = [lo[0] + d[0] + 3, mid[1], mid[2]]
            for c in range(3):
                s["idx"][c][_ellipsoid(n, c, at, [5.0] * 3)] = len(s["materials"]) - 1
        i, j, k = s["sources"][0]["i"], s["sources"][0]["j"], s["sources"][0]["k"]
        for c in range(3):                            # the dipole sits in vacuum
            s["idx"][c][i - 1:i + 2, j - 1:j + 2, k - 1:k + 2] = 0
    if s["idx"] is not None:
        s["idx"] = [a.to(torch.uint8) for a in s["idx"]]
    return s


def _initial(s, seed, comp, which=0):
    """Component comp of a field in progress: three travelling waves of 14 to 50 cells under a window that is zero in the absorbers."""
    rng = np.random.default_rng([seed, which, comp, 77])
    out = torch.zeros(s["n"], dtype=torch.float32, device="cuda")
    x = [torch.arange(m, dtype=torch.float32, device="cuda") for m in s["n"]]
    for _ in range(3):
        k = rng.normal(size=3)
        k *= 2 * math.pi / rng.uniform(14.0, 50.0) / np.linalg.norm(k)
        arg = (float(k[0]) * x[0] + float(rng.uniform(0, 6.28)))[:, None, None] + (float(k[1]) * x[1])[:, None] + float(k[2]) * x[2]
        out += torch.sin_(arg)
    lo = (16, 16, 4) if s["geometry"] == "reference" else [p[0] + 1 if p[0] else 0 for p in s["pml"]]
    hi = (16, 16, 17) if s["geometry"] == "reference" else [p[1] + 1 if p[1] else 0 for p in s["pml"]]
    for a, m in enumerate(s["n"]):
        u = ((x[a] - lo[a]) / (m - 1 - hi[a] - lo[a])).clamp(0.0, 1.0)
        out *= torch.sin(math.pi * u).square().reshape([-1 if b == a else 1 for b in range(3)])
    if s["tfsf"] is None:
        return out
    return out.mul_(0.2)                              # the incident pulse on top of what has been scattered


# ------------------------------------------------------------------ the framework's side
class _Device:
    """A device array of a Simulation, which lives as long as a tensor on it does."""

    def __init__(self, sim, ptr, shape, strides):
        self.sim = sim
        self.__cuda_array_interface__ = dict(shape=tuple(shape), strides=tuple(4 * v for v in strides), typestr="<f4",
                                             data=(ptr, False), version=3)


def _view(sim, comp):
    """The engine's current array of one component, in place on the device."""
    ptr, strides = sim.device_ptr(comp)
    return torch.as_tensor(_Device(sim, ptr, sim.shape, strides), device="cuda")


def _on_device(case):
    """Large runs keep their fields on the device; small ones are read through host arrays."""
    return case["engine"] == "tuned" or case["order"] == 4


def _simulation(case, seed, which=0):
    s = _setup(case, seed, which)
    n = s["n"]
    geometry = dict(box=abi.GEOM_BOX, reference=abi.GEOM_REFERENCE)[s["geometry"]]
    absorber = dict(none=abi.ABS_NONE, cpml=abi.ABS_CPML, split=abi.ABS_SPLIT_PML)[s["absorber"]]
    sim = Simulation(abi.make_config(*n, dx=s["ds"], dt=s["dt"], order=s["order"], geometry=geometry, absorber=absorber, pml=s["pml"],
                                     spml_vmax=s.get("vmax", 1.0), probe_every=s["every"], probe_capacity=s["steps"] // s["every"]))
    table = []
    for m in s["materials"]:
        if "poles" in m:
            table.append(abi.make_material(1.0, poles=m["poles"], eps_inf=m["eps_inf"], sigma=m["sigma"]))
        elif "gyro" in m:
            table.append(abi.make_material(1.0, eps_inf=m["eps_inf"], gyro=m["gyro"]))
        else:
            table.append(abi.make_material(m["eps"]))
    if s["idx"] is not None:
        sim.set_materials(table, *[a.cpu().numpy() for a in s["idx"]])
    for q in s["sources"]:
        sim.add_point_source(abi.PointSource(comp=q["comp"], i=q["i"], j=q["j"], k=q["k"], waveform=abi.WAVE_GAUSS_SINE, amp=q["amp"],
                                             f0=q["f0"], tau=q["tau"], t0=q["t0"]))
    t = s["tfsf"]
    if t is not None:
        src = abi.TFSF()
        src.kind = abi.TFSF_PLANE_X if t["kind"] == "plane" else abi.TFSF_DIPOLE
        src.box_lo[:], src.box_hi[:] = t["lo"], t["hi"]
        src.ntime = s["every"]
        for key in ("amp", "f0", "tau", "t0", "c", "w", "kenv"):
            if key in t:
                setattr(src, key, t[key])
        sim.set_tfsf(src)
    for c, i, j, k, mode in s["probes"]:
        sim.add_probe(c, i, j, k, abi.PROBE_REFERENCE if mode else abi.PROBE_NODE)
    planes = [sim.add_dft_plane(axis, index, sum(1 << c for c in comps), om) for axis, index, comps, om in s["dft"]]
    boxes = [sim.add_flux_box(lo, hi, om) for lo, hi, om in s["flux"]]
    if s["design"] is not None:
        sim.set_design(*s["design"])
    for c in range(6):
        f = _initial(s, seed, c, which)
        if _on_device(case) and s["geometry"] == "box":
            _view(sim, c).copy_(f)
        else:
            sim.set_field(c, f.cpu().numpy())
    torch.cuda.synchronize()
    if case["engine"] == "tuned":
        sim.autotune(12)
    elif case["engine"] == "sweep":
        sim.set_engine(3)
    return s, sim, planes, boxes


def prepare(case, seed):
    if case["kind"] != "gradient":
        s, sim, planes, boxes = _simulation(case, seed)
        return dict(case=case, sim=sim, planes=planes, boxes=boxes)
    made = [_simulation(case, seed, w) for w in range(case["count"])]
    if not case["history"]:
        for _, sim, _, _ in made:
            sim.set_adjoint_memory(0)
    return dict(case=case, sims=[m[1] for m in made], plane_x=[m[0]["plane_x"] for m in made], omega=[m[0]["omega"] for m in made])


def run(state):
    case = state["case"]
    if case["kind"] == "gradient":
        if case["count"] == 1:
            j, grad = state["sims"][0].forward_adjoint(case["steps"], state["plane_x"][0], state["omega"][0], 25)
            return dict(objective=[j], gradient=[grad])
        j, grad = batch_forward_adjoint(state["sims"], case["steps"], state["plane_x"], state["omega"], 25)
        return dict(objective=j, gradient=grad)
    sim = state["sim"]
    sim.step(case["steps"])
    out = dict(traces=sim.read_probes(), spectra=[sim.read_dft(p) for p in state["planes"]], flux=[sim.read_flux(b)[0] for b in state["boxes"]])
    if _on_device(case):
        out["fields"] = [_view(sim, c) for c in range(6)]
    else:
        out["fields"] = [sim.get_field(c) for c in ((EZ, HY) if case["nx"] * case["ny"] * case["nz"] > 1e6 else range(6))]
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Per time step each field is read and written once (48 bytes a cell) with the absorber's auxiliaries in its cells, the state of
    dispersive nodes and the material indices; the adjoint of a step does the same once more.  About 36 operations a cell."""
    count = case.get("count", 1)
    n = (case["nx"], case["ny"], case["nz"])
    cells = float(n[0] * n[1] * n[2])
    pml = case["pml"]
    slab = sum(2 * pml * cells / m for m in n)
    if case["kind"] == "reference":
        slab = 30 * cells / n[0] + 30 * cells / n[1] + 16 * cells / n[2]
    small = min(n)
    disp = {"lorentz": 4 / 3 * math.pi * 0.008 * cells * 10, "drude_tfsf": 4 / 3 * math.pi * (0.104 * small) ** 3 * 6,
            "reference": 8 / n[2] * cells * 6, "gyro": 0.2 * cells * 2}.get(case["kind"], 0.0)   # words of state a node keeps
    per_step = 48 * cells + 32 * slab + 3 * 8 * disp
    ops = 36.0 * cells if case["order"] == 2 else 60.0 * cells
    if case["kind"] == "drude_tfsf":
        plane = 4.0 * n[1] * n[2]
        per_step += 4 * plane + 2 * 16 * 16 * plane / 16       # samples; the spectra once in 16 steps
        ops += 4 * 16 * plane
    if case["kind"] == "gradient":
        d = 3.0 * case["design"] ** 3 / 2
        return dict(bytes=count * case["steps"] * (2 * per_step + 4 * d * 4), flops=count * case["steps"] * 2 * ops)
    return dict(bytes=case["steps"] * per_step, flops=case["steps"] * ops)


def tolerance(case):
    # about four times the 32-bit rounding seen against exact()
    if case["kind"] in ("drude_tfsf", "reference"):
        # a Drude current is integrated twice over time, and its rounding with it: up to 6e-5 of a field after 200 steps
        return {"rel": 2.5e-4, "max": 2.5e-2}
    return {"rel": 1e-5, "max": 1e-3}


# ------------------------------------------------------------------ the same equations in plain torch, 64 bits
def _offset(comp, axis):
    """Half-cell offset of a component's nodes along an axis."""
    return int(axis != comp) if comp < 3 else int(axis == comp - 3)


def _along(v, axis):
    return v.reshape([-1 if b == axis else 1 for b in range(3)])


class _Plain:
    """Leapfrog H then E; every array is replaced, never changed in place, so that torch can differentiate through it."""

    def __init__(self, s, seed, which=0, ie_design=None):
        self.s, n = s, s["n"]
        f64 = dict(dtype=torch.float64, device="cuda")
        self.f = [_initial(s, seed, c, which).double() for c in range(6)]
        self.cdt = s["dt"] / s["ds"]
        eps = torch.ones(len(s["materials"]), 3, **f64)
        for m, d in enumerate(s["materials"]):
            e = d.get("eps", d.get("eps_inf"))
            eps[m] = torch.tensor([e] * 3 if isinstance(e, float) else list(e), **f64)
        self.single = s["idx"] is None
        self.ie = [torch.ones(1, 1, 1, **f64) if self.single else (1.0 / eps[:, c])[s["idx"][c].long()] for c in range(3)]
        if ie_design is not None:
            lo, d = s["design"][0], s["design"][1].shape[1:]
            box = tuple(slice(lo[a], lo[a] + d[a]) for a in range(3))
            for c in range(3):
                full = self.ie[c].clone()
                full[box] = ie_design[c]
                self.ie[c] = full
        # live index ranges and the rule outside them
        self.live, self.rule = {}, {}
        for c in range(6):
            for a in range(3):
                o, m = _offset(c, a), n[a]
                lo, hi, rule = 0, m - 1, (None, None)
                if s["geometry"] == "reference":
                    if a == 0:
                        ok = [v for v in range(m) if 3 < 2 * v + o < 2 * m - 3]
                    else:
                        top = 2 * m - 3 if a == 1 else 2 * m - 1
                        ok = [v for v in range(m) if 2 * v + o <= top]
                        rule = ((0, -1.0 if a == 1 and c >= 3 else 1.0), (top, 1.0))
                    lo, hi = ok[0], ok[-1]
                self.live[c, a], self.rule[c, a] = (lo, hi), rule
        self.pick = {}
        if s["geometry"] == "reference":
            for c in range(6):
                for a in range(3):
                    lo, hi = self.live[c, a]
                    keep = torch.zeros(n[a], **f64)
                    keep[lo:hi + 1] = 1.0
                    self.f[c] = self.f[c] * _along(keep, a)
        self._absorber()
        self._dispersion()
        g = [m.get("gyro") for m in s["materials"]]
        self.gyro = None
        if any(g):
            dt = s["dt"]
            col = torch.tensor([[0.0] * 5 if q is None else [math.exp(-q[1] * dt), math.cos(q[2] * dt), math.sin(q[2] * dt), q[0] ** 2 * dt,
                                                             dt / s["materials"][m]["eps_inf"]] for m, q in enumerate(g)], **f64)
            self.gyro = [[col[:, v][s["idx"][c].long()] for v in range(5)] for c in range(3)]
            self.J = [torch.zeros(n, **f64) for _ in range(3)]
        self.step_no = 0
        self.traces = [[] for _ in s["probes"]]
        self.sums = [[[torch.zeros((), dtype=torch.complex128, device="cuda") for _ in om] for _ in comps] for _, _, comps, om in s["dft"]]
        self.faces = []
        for lo, hi, om in s["flux"]:
            for a in range(3):
                comps = ((a + 1) % 3, (a + 2) % 3, 3 + (a + 1) % 3, 3 + (a + 2) % 3)
                for at in (lo[a], hi[a]):
                    self.faces.append((a, at, lo, hi, comps, om, [[0.0 for _ in om] for _ in comps]))
        if s["tfsf"] is not None:
            self._box()

    # -- absorber: per (component, axis, side) the coefficients over the slab and the auxiliary values
    def _absorber(self):
        s, n = self.s, self.s["n"]
        self.slabs, self.aux = {}, {}
        if s["absorber"] == "none":
            return
        dt, ds = s["dt"], s["ds"]
        for a in range(3):
            for side in range(2):
                depth = s["pml"][a][side]
                if not depth:
                    continue
                first = 0 if side == 0 else n[a] - depth
                for c in range(6):
                    if (c % 3) == a:
                        continue
                    p, q = [], []
                    for v in range(first, first + depth):
                        h = 2 * v + _offset(c, a)
                        if s["absorber"] == "cpml":
                            dep = min(float(depth), (2 * depth - 1 - h) / 2 if side == 0 else (h - (2 * n[a] - 2 * depth)) / 2)
                            sg = 0.8 * 4.0 / ds * (max(dep, 0.0) / depth) ** 3
                            b = math.exp(-sg * dt)
                            p.append(b)
                            q.append(b - 1.0 if sg > 0 else 0.0)
                        else:
                            k2 = self._split_k2(a, h)
                            p.append(2 * k2 - 1)
                            q.append(k2)
                    f64 = dict(dtype=torch.float64, device="cuda")
                    self.slabs.setdefault((c, a), []).append((first, depth, _along(torch.tensor(p, **f64), a), _along(torch.tensor(q, **f64), a)))
                    self.aux[c, a, first] = 0.0

    def _split_k2(self, a, h):
        """Damping of the split-field layer at half-coordinate h (quartic grading, tables of 4 halves a cell)."""
        s = self.s
        n, dt, ds, vmax = s["n"][a], s["dt"], s["ds"], s["vmax"]
        size = 4 * (s["pml"][a][0] if a < 2 else s["pml"][2][1])

        def gamma(i, big):
            if i >= big - 3:
                return 0.0
            i, big = max(i, 0), big - 3
            top = (vmax * math.log(10000.0) * 5.0 / (2.0 * big * ds * 0.5)) ** 0.25
            return (top - i * top / big) ** 4
        if a == 0:
            edge = 2 * s["pml"][0][0] - 3
            i = h if h < edge else h - 2 * n + size if h >= 2 * n - edge else None
            g = None if i is None else gamma(size // 2 - abs(i - size // 2) - 3, size // 2 - 3)
        elif a == 1:
            i = h if h < size // 2 else h - 2 * n + size if h >= 2 * n - size // 2 else None
            g = None if i is None else gamma(i if i < size // 2 else size - i - 3, size // 2)
        else:
            i = h - 2 * n + size
            g = gamma(size - i - 1, size // 2) if size // 2 <= i < size else None
        return 1.0 if g is None else 1.0 / (1.0 + 0.5 * dt * g)

    def _dispersion(self):
        s, dt = self.s, self.s["dt"]
        self.disp = []
        for m, d in enumerate(s["materials"]):
            if "poles" not in d:
                continue
            co, zp, zm, zz = [], 0.0, 0.0, 0.0
            for k, deps, wp, gp, gq in d["poles"]:
                a0, a1, b0, b1 = deps * wp * wp, deps * gq, 0.0 if k == 1 else wp * wp, 2 * gp
                den = b1 * dt + 2
                r = ((4 - 2 * b0 * dt * dt) / den, (b1 * dt - 2) / den, (a0 * dt * dt + 2 * a1 * dt) / den, (2 * a1 * dt - a0 * dt * dt) / den,
                     -4 * a1 * dt / den)
                zp, zm, zz = zp + r[2], zm + r[3], zz + r[4]
                co.append(r)
            den = 2 * d["eps_inf"] + d["sigma"] * dt + zp
            top = (-zm / den, (2 * d["eps_inf"] - d["sigma"] * dt - zz) / den, 2 * dt / den)
            for c in range(3):
                at = torch.nonzero(s["idx"][c].flatten() == m).flatten()
                if s["geometry"] == "reference":      # nodes held at zero stay there
                    sub = torch.ones(s["n"], dtype=torch.bool, device="cuda")
                    for a in range(3):
                        lo, hi = self.live[c, a]
                        v = torch.arange(s["n"][a], device="cuda")
                        sub &= _along((v >= lo) & (v <= hi), a)
                    at = at[sub.flatten()[at]]
                zero = torch.zeros(len(at), dtype=torch.float64, device="cuda")
                self.disp.append(dict(c=c, at=at, co=co, top=top, em=zero, jp=[zero] * len(co), jm=[zero] * len(co)))

    def _tap(self, c, a, o):
        """Component c shifted by o nodes along a, by the boundary's rule."""
        n, f = self.s["n"][a], self.f[c]
        if self.rule[c, a] == (None, None):
            pad = [0, 0] * (2 - a) + ([0, o] if o > 0 else [-o, 0])
            return f if o == 0 else torch.nn.functional.pad(f.narrow(a, max(o, 0), n - abs(o)), pad)
        key = (c, a, o)
        if key not in self.pick:
            at, sign = [], []
            lo, hi = self.live[c, a]
            for v in range(o, n + o):
                w, g = v, 1.0
                if v < lo or v > hi:
                    plane, g = self.rule[c, a][0 if v < lo else 1]
                    w = plane - v - _offset(c, a)
                    if w < lo or w > hi:
                        w, g = 0, 0.0
                at.append(w)
                sign.append(g)
            self.pick[key] = (torch.tensor(at, device="cuda"), _along(torch.tensor(sign, dtype=torch.float64, device="cuda"), a))
        at, sign = self.pick[key]
        return f.index_select(a, at) * sign

    def _taps(self, c):
        at = (-1, 0) if c >= 3 else (0, 1)
        return list(zip(at, (-1.0, 1.0))) if self.s["order"] == 2 else list(zip((at[0] - 1, *at, at[1] + 1), (1 / 24, -27 / 24, 27 / 24, -1 / 24)))

    def _terms(self, c):
        """The two curl terms of component c: (axis, source component, sign)."""
        a, b = (c + 1) % 3, (c + 2) % 3
        o, sg = (3, 1.0) if c < 3 else (0, -1.0)
        return (a, o + b, sg), (b, o + a, -sg)

    def _box(self):
        """Index ranges of the total-field box and, per curl term, the taps that cross its surface."""
        s, t, n = self.s, self.s["tfsf"], self.s["n"]
        inside = [[h for h in range(2 * n[a] + 2) if t["lo"][a] < 0.5 * h * s["ds"] < t["hi"][a]] for a in range(3)]
        lo, hi = [v[0] for v in inside], [v[-1] for v in inside]
        self.lo = lo
        self.cross = {}
        for c in range(6):
            for a, g, sg in self._terms(c):
                if t["kind"] == "plane" and g not in (EZ, HY):
                    continue
                rows = []
                for o, w in self._taps(c):
                    for v in range(n[a]):
                        mine, other = 2 * v + _offset(c, a), 2 * (v + o) + _offset(g, a)
                        if (lo[a] <= mine <= hi[a]) != (lo[a] <= other <= hi[a]):
                            rows.append((v, v + o, w * (-1.0 if lo[a] <= mine <= hi[a] else 1.0)))
                rng = [[v for v in range(n[b]) if lo[b] <= 2 * v + _offset(g, b) <= hi[b]] for b in range(3)]
                self.cross.setdefault(c, []).append((a, g, sg, rows, [(r[0], r[-1] + 1) for r in rng]))
        if t["kind"] == "plane":
            self.pad = 600
            self.le = torch.zeros(n[0] + 2 * self.pad, dtype=torch.float64, device="cuda")
            self.lh = torch.zeros_like(self.le)
            self.at = (lo[0] - 1) // 2 - 10 + self.pad

    def _incident(self, g, x, y, z, tt):
        """Field of a z dipole under a Hann-windowed sine, at whole arrays of positions (physical units), time tt steps."""
        t = self.s["tfsf"]
        c, w, ke = t["c"], t["w"], t["kenv"]
        ctr = [0.5 * (t["lo"][a] + t["hi"][a]) for a in range(3)]
        x, y, z = x - ctr[0], y - ctr[1], z - ctr[2]
        r = torch.sqrt(x * x + y * y + z * z)
        ph = w * (tt * self.s["dt"] - r / c)
        env, denv, ddenv = 0.5 * (1 - torch.cos(ke * ph)), 0.5 * w * ke * torch.sin(ke * ph), 0.5 * (w * ke) ** 2 * torch.cos(ke * ph)
        sn, cs = torch.sin(ph), torch.cos(ph)
        on = ((ph >= 0) & (ke * ph <= 2 * math.pi)).double()
        d, d1, d2 = on * sn * env, on * (w * cs * env + sn * denv), on * (-w * w * sn * env + 2 * w * cs * denv + sn * ddenv)
        ux, uy, uz = x / r, y / r, z / r
        if g < 3:
            u = (ux, uy, uz)[g]
            e = 1.0 if g == 2 else 0.0
            far = d2 * (uz * u - e)
            return c * (far / (c * c * r) + (3 * uz * u - e) * d1 / (c * r * r) + (3 * uz * u - e) * d / r ** 3)
        u = -uy if g == 3 else ux if g == 4 else 0.0 * ux
        return u * (d2 / (c * c * r) + d1 / (c * r * r))

    def _correct(self, c, new, tt):
        s, t = self.s, self.s["tfsf"]
        for a, g, sg, rows, rng in self.cross.get(c, ()):
            for v, tap, w in rows:
                box = [slice(*r) for r in rng]
                box[a] = slice(v, v + 1)
                if t["kind"] == "plane":
                    line = self.le if g == EZ else self.lh
                    if a == 0:
                        inc = line[tap + self.pad].reshape(1, 1, 1)
                    else:
                        inc = line[rng[0][0] + self.pad: rng[0][1] + self.pad].reshape(-1, 1, 1)
                else:
                    pos = []
                    for b in range(3):
                        i = torch.arange(*(rng[b] if b != a else (tap, tap + 1)), dtype=torch.float64, device="cuda")
                        pos.append(_along((i + 0.5 * _offset(g, b)) * s["ds"], b))
                    inc = self._incident(g, *pos, tt)
                ie = 1.0 if c >= 3 else self.ie[c] if self.ie[c].numel() == 1 else self.ie[c][tuple(box)]
                new[tuple(box)] += ie * sg * self.cdt * w * inc
        return new

    def _line(self, f, taps):
        out = torch.zeros_like(f)
        for o, w in taps:
            m = len(f) - abs(o)
            out[max(-o, 0): max(-o, 0) + m] += w * f[max(o, 0): max(o, 0) + m]
        return self.cdt * out

    def _half(self, comps, tt):
        fresh = {}
        for c in comps:
            total = None
            raw = []
            for a, g, sg in self._terms(c):
                d = None
                for o, w in self._taps(c):
                    v = self._tap(g, a, o)
                    d = v * (w * sg * self.cdt) if d is None else d.add(v, alpha=w * sg * self.cdt)
                raw.append(d)
                for first, depth, p, q in self.slabs.get((c, a), ()):
                    key = (c, a, first)
                    part, old = d.narrow(a, first, depth), self.aux[key]
                    new = p * old + q * part
                    self.aux[key] = new
                    parts = [d.narrow(a, 0, first), part + new if self.s["absorber"] == "cpml" else new - old,
                             d.narrow(a, first + depth, d.shape[a] - first - depth)]
                    d = torch.cat(parts, dim=a)
                total = d if total is None else total + d
            if c < 3:
                new = self.f[c] + self.ie[c] * total
                for m in self.disp:
                    if m["c"] == c and len(m["at"]):
                        new = self._ade(m, c, new, (raw[0] + raw[1]).flatten()[m["at"]])
                if self.gyro is not None:
                    new = new - self.gyro[c][4] * self.J[c]
            else:
                new = self.f[c] + total
            if self.s["geometry"] == "reference":
                for a in range(3):
                    lo, hi = self.live[c, a]
                    new = torch.nn.functional.pad(new.narrow(a, lo, hi + 1 - lo), [0, 0] * (2 - a) + [lo, self.s["n"][a] - 1 - hi])
            fresh[c] = new
        for c in comps:
            q = self.step_no
            for p in self.s["sources"]:
                if p["comp"] == c:
                    u = (q + 0.5) * self.s["dt"] - p["t0"]
                    fresh[c][p["i"], p["j"], p["k"]] += p["amp"] * math.sin(2 * math.pi * p["f0"] * u) * math.exp(-(u / p["tau"]) ** 2)
            self.f[c] = self._correct(c, fresh[c], tt) if self.s["tfsf"] is not None else fresh[c]

    def _ade(self, m, c, new, rot):
        (c1, c2, c3), e, em = m["top"], self.f[c].flatten()[m["at"]], m["em"]
        out = c1 * em + c2 * e + c3 / self.s["dt"] * rot
        for (al, xi, _, _, _), jp, jm in zip(m["co"], m["jp"], m["jm"]):
            out = out - 0.5 * c3 * ((1 + al) * jp + xi * jm)
        dt = self.s["dt"]
        fresh = [al * jp + xi * jm + (zp * out + zm * em + z0 * e) / dt for (al, xi, zp, zm, z0), jp, jm in zip(m["co"], m["jp"], m["jm"])]
        m["jm"], m["jp"], m["em"] = m["jp"], fresh, e
        return new.flatten().index_copy(0, m["at"], out).reshape(new.shape)

    def _current(self):
        def shift(v, a, o):
            pad = [0, 0] * (2 - a) + ([0, o] if o > 0 else [-o, 0])
            return torch.nn.functional.pad(v.narrow(a, max(o, 0), v.shape[a] - abs(o)), pad)
        x, y, z = self.J
        ym, xm = shift(y, 0, -1), shift(x, 1, -1)
        ay = 0.25 * (y + ym + shift(y, 1, 1) + shift(ym, 1, 1))
        ax = 0.25 * (x + xm + shift(x, 0, 1) + shift(xm, 0, 1))
        g = self.gyro
        self.J = [(g[0][1] * x + g[0][2] * ay) * g[0][0] + g[0][3] * self.f[0], (g[1][1] * y - g[1][2] * ax) * g[1][0] + g[1][3] * self.f[1],
                  g[2][0] * z + g[2][3] * self.f[2]]

    def step(self):
        s, q = self.s, self.step_no
        plane = s["tfsf"] is not None and s["tfsf"]["kind"] == "plane"
        self._half((3, 4, 5), float(q))
        if plane:
            self.lh = self.lh + self._line(self.le, self._taps(HX))
        if self.gyro is not None:
            self._current()
        self._half((0, 1, 2), q + 0.5)
        if plane:
            t = s["tfsf"]
            self.le = self.le + self._line(self.lh, self._taps(EX))
            u = (q + 0.5) * s["dt"] - t["t0"]
            self.le[self.at] += t["amp"] * math.sin(2 * math.pi * t["f0"] * u) * math.exp(-(u / t["tau"]) ** 2)
        self.step_no = q = q + 1
        if q % s["every"] == 0:
            for tr, p in zip(self.traces, s["probes"]):
                tr.append(self._probe(*p))
        for (axis, index, comps, om), acc in zip(s["dft"], self.sums):
            for c, row in zip(comps, acc):
                v = self.f[c].select(axis, index)
                for k, w in enumerate(om):
                    row[k] = row[k] + v * self._phase(c, w)
        for a, at, lo, hi, comps, om, acc in self.faces:
            b, c = [v for v in range(3) if v != a]
            for comp, row in zip(comps, acc):
                v = self.f[comp].select(a, at)[lo[b]:hi[b], lo[c]:hi[c]]
                for k, w in enumerate(om):
                    row[k] = row[k] + v * self._phase(comp, w)

    def _phase(self, c, w):
        a = w * (self.step_no - (0.5 if c >= 3 else 0.0)) * self.s["dt"]
        return complex(math.cos(a), -math.sin(a)) * self.s["dt"]

    def _probe(self, c, i, j, k, mode):
        f = self.f[c]
        if not mode:
            return f[i, j, k]
        km = k - 1 if k else 1
        if c == 0:
            return (f[i, j - 1, km] + f[i, j - 1, k] + f[i, j, km] + f[i, j, k]) / 4
        if c == 1:
            return (f[i - 1, j, km] + f[i - 1, j, k] + f[i, j, km] + f[i, j, k]) / 4
        if c == 2:
            return (f[i - 1, j - 1, k] + f[i - 1, j, k] + f[i, j - 1, k] + f[i, j, k]) / 4
        if c == 3:
            return (f[i - 1, j, k] + f[i, j, k]) / 2
        if c == 4:
            return (f[i, j - 1, k] + f[i, j, k]) / 2
        return f[i, j, km] / 2                        # one of the two points the sensor averages is never set

    def flux(self):
        out = []
        for q, (a, at, lo, hi, comps, om, acc) in enumerate(self.faces):
            sign = -1.0 if q % 2 == 0 else 1.0
            out.append([sign * float((acc[0][k] * acc[3][k].conj() - acc[1][k] * acc[2][k].conj()).real.sum()) for k in range(len(om))])
        return out


def _exact_gradient(case, seed, which):
    s = _setup(case, seed, which)
    ie = (1.0 / torch.tensor(s["design"][1], dtype=torch.float64, device="cuda")).requires_grad_(True)
    p = _Plain(s, seed, which, ie)
    sums = {c: 0.0 for c in (EY, EZ, HY, HZ)}
    for _ in range(s["steps"]):
        p.step()
        for c in sums:
            sums[c] = sums[c] + p.f[c][s["plane_x"]] * p._phase(c, s["omega"])
    j = (sums[EY] * sums[HZ].conj() - sums[EZ] * sums[HY].conj()).real.sum()
    j.backward()
    return float(j.detach()), (-(ie * ie) * ie.grad).detach()


def exact(case, seed):
    if case["kind"] == "gradient":
        if case["count"] * case["steps"] * case["nx"] * case["ny"] * case["nz"] > 6e8:
            return None
        got = [_exact_gradient(case, seed, w) for w in range(case["count"])]
        return dict(objective=[g[0] for g in got], gradient=[g[1] for g in got])
    s = _setup(case, seed)
    p = _Plain(s, seed)
    with torch.no_grad():
        for _ in range(s["steps"]):
            p.step()
    traces = torch.stack([torch.stack(t) for t in p.traces])
    spectra = [torch.stack([torch.stack(row) for row in acc]).cpu().numpy() for acc in p.sums]
    out = dict(traces=traces, spectra=spectra, flux=[np.array(p.flux())] if p.faces else [])
    if _on_device(case):
        out["fields"] = p.f
    else:
        out["fields"] = [p.f[c] for c in ((EZ, HY) if case["nx"] * case["ny"] * case["nz"] > 1e6 else range(6))]
    return out
