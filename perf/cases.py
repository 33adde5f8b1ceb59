"""Performance cases: what a program built on this library spends its time on.

Every case goes through the public entry points (``capi.Lattice``,
``batch.Batch``, ``driver.cluster_stats`` and the C ABI behind them).  Five
kinds of work:

* ``steps``    a time loop that advances a resident lattice by ``steps`` and
               takes the density field (and, with ``velocity``, the velocity
               field) off it, device to device;
* ``job``      a whole small job: host geometry and density in, initialise,
               ``steps`` time steps, the density field back on the host;
* ``batch``    many independent domains of uneven size advanced together, the
               density field of each taken off;
* ``stats``    the phase statistics and the per-plane profile of a lattice;
* ``clusters`` the cluster statistics of a two-phase field (host arrays in,
               labels and the statistics row out).

Lattices are sphere packings as the benchmarks use them.  ``drainage`` holds
an inlet slab at a low density and an outlet plane at a high one in a packing
filled with liquid; without it the box is periodic and the density starts
with a small perturbation.  G = -5 for drainage: the coupling at which a long
run stays finite.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from multiphase_lbm_b200 import batch, capi, driver, host

STORAGE = {"f32": capi.STORE_F32, "f16": capi.STORE_F16, "f64": capi.STORE_F64}
RHO_L, RHO_G = 0.2726, 0.0484  # default spinodal densities


def _case(name, **kw):
    c = dict(kind="steps", nx=64, ny=64, nz=64, storage="f32", porosity=0.5,
             rmin=2.5, rmax=7.5, drainage=False, tau=1.0, G=-6.0,
             carn_star=False, inject=False, velocity=False, steps=10)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: one step of a small box and its density, the
        # loop of a program that looks at every step
        _case("step_32_f32", nx=32, ny=32, nz=32, steps=1),
        # phase separation in a small periodic box (the 64^3 configuration),
        # long runs of steps between looks
        _case("periodic_64_f32", steps=50),
        # the headline: 200^3 drainage, ten steps (the default statistics
        # period) between looks
        _case("drainage_200_f32", nx=200, ny=200, nz=200, rmin=5.0, rmax=15.0,
              drainage=True, G=-5.0),
        # the largest: the 384^3 precision configuration in FP16 storage
        _case("drainage_384_f16", nx=384, ny=384, nz=384, rmin=5.0, rmax=15.0,
              drainage=True, G=-5.0, storage="f16", steps=4),
        # odd edges, no alignment anywhere, velocity output
        _case("ragged_f32_velocity", nx=193, ny=77, nz=131, velocity=True),
        # FP64: the runs other storages are judged against
        _case("drainage_96_f64", nx=96, ny=96, nz=96, storage="f64",
              drainage=True, G=-5.0),
        # a relaxation time other than 1
        _case("tau08_160_f32", nx=160, ny=144, nz=128, rmin=4.0, rmax=10.0,
              drainage=True, G=-5.0, tau=0.8),
        # Carnahan-Starling equation of state with density injection
        _case("cs_inject_f32", nx=97, ny=65, nz=81, carn_star=True, G=-1.0,
              inject=True),
        # a served mix: uneven domains in FP16 storage, advanced together
        _case("batch_48_f16", kind="batch", nx=128, ny=48, nz=0, drainage=True,
              G=-5.0, storage="f16", steps=6),
        # a short job from host arrays to host arrays
        _case("job_128_f32", kind="job", nx=128, ny=128, nz=128, drainage=True,
              G=-5.0, steps=20),
        # statistics of a running 200^3 lattice
        _case("stats_200_f32", kind="stats", nx=200, ny=200, nz=200, rmin=5.0,
              rmax=15.0, drainage=True, G=-5.0),
        # the cluster columns of a statistics row
        _case("clusters_128", kind="clusters", nx=128, ny=128, nz=128),
    ]


def draw(rng):
    """One more case of the same ranges: boxes of 24 to about 320 nodes an
    edge (odd ones among them), every storage, boundary and option."""
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choices(["steps", "job", "batch", "stats", "clusters"],
                       [12, 2, 2, 2, 2])[0]
    storage = rng.choices(["f32", "f16", "f64"], [5, 3, 2])[0]
    big = {"steps": 320, "job": 192, "batch": 128, "stats": 320,
           "clusters": 160}[kind]
    if storage == "f64":
        big = min(big, 160)
    c = _case(None, kind=kind, storage=storage, nx=edge(24, big),
              ny=edge(24, big), nz=edge(24, big),
              porosity=round(rng.uniform(0.35, 0.75), 3),
              drainage=rng.random() < 0.6)
    if min(c["nx"], c["ny"], c["nz"]) > 60 and rng.random() < 0.5:
        c.update(rmin=5.0, rmax=15.0)
    c["G"] = -5.0 if c["drainage"] else -6.0
    if rng.random() < 0.25:
        c["tau"] = round(rng.uniform(0.7, 1.3), 2)
    if not c["drainage"] and rng.random() < 0.2:
        c.update(carn_star=True, G=-1.0)
    if rng.random() < 0.15:
        c["inject"] = True
    c["velocity"] = kind == "steps" and storage != "f16" and rng.random() < 0.4
    most = 6 if storage == "f16" else 50
    nodes = c["nx"] * c["ny"] * c["nz"]
    c["steps"] = rng.randint(1, max(1, min(most, int(1.5e8 / nodes))))
    if kind == "batch":
        # nx: the largest edge of a domain, ny: the number of domains
        c.update(nx=rng.randint(48, 128), ny=rng.randint(8, 60), nz=0,
                 carn_star=False, G=-5.0, drainage=True,
                 steps=rng.randint(1, 6))
    if kind == "clusters":
        c.update(storage="f32")
    return c


# ---- inputs -----------------------------------------------------------------

def _params(c, shape, **kw):
    p = dict(G=c["G"], tau=c["tau"], rho_shift=1.0)
    if c["carn_star"]:
        p.update(carn_star=1, T_Tc=0.7, rhos=0.35)
    else:
        p.update(rhos=-math.log(1.0 + 1.0 / c["G"]))  # G_ads = -1
    if c["drainage"]:
        p.update(inlet_width=max(1, round(8 * shape[0] / 200)),
                 outlet_width=1, rho_inlet=0.10, rho_outlet=1.95)
    p.update(rho_increment=1e-5 if c["inject"] else 0.0,
             rho_inject_period=3 if c["inject"] else 0,
             inject_position=0.5, inject_density=1 if c["inject"] else 0)
    p.update(kw)
    return capi.default_params(**p)


def _density(c, shape, rng):
    if c["drainage"]:
        return np.full(shape, 2.0, np.float32)
    base, amp = (0.2, 0.01) if c["carn_star"] else (0.70, 0.01)
    return (base - amp + 2 * amp * rng.random(shape, np.float32)).astype(np.float32)


def _domains(c, seed):
    """[(shape, fluid, rho, params)] of a case: one lattice, or a batch's."""
    if c["kind"] != "batch":
        shape = (c["nx"], c["ny"], c["nz"])
        fluid, _ = host.generate_packing(shape, c["rmin"], c["rmax"],
                                         c["porosity"], seed, device=_device())
        return [(shape, fluid, _density(c, shape, np.random.default_rng(seed)),
                 _params(c, shape))]
    rng = np.random.default_rng(c["ny"])  # the mix of sizes is the case's
    edges = np.arange(32, c["nx"] + 1, 16)
    out = []
    for i in range(c["ny"]):
        shape = tuple(int(v) for v in rng.choice(edges, 3))
        por = float(rng.uniform(0.35, 0.65))
        gads = float(rng.uniform(-2.0, 0.0))
        fluid, _ = host.generate_packing(shape, c["rmin"], c["rmax"], por,
                                         seed * 1009 + i, device=_device())
        out.append((shape, fluid,
                    _density(c, shape, np.random.default_rng(seed)),
                    _params(c, shape, rhos=-math.log(1.0 - gads / c["G"]))))
    return out


def _device():
    return 0 if torch.cuda.is_available() else None


def _field_tensors(c, shapes):
    kind = torch.float64 if c["storage"] == "f64" else torch.float32
    return [torch.empty(s, dtype=kind, device="cuda") for s in shapes]


def _lattice(c, shape, fluid, rho, params):
    lat = capi.Lattice(shape, storage=STORAGE[c["storage"]])
    lat.set_params(params)
    lat.upload(fluid, rho)
    lat.initialize()
    return lat


def _two_phase(c, seed):
    """A packing with numbered grains and a smooth density field with liquid
    and vapour regions, as a run leaves it."""
    shape = (c["nx"], c["ny"], c["nz"])
    _, spheres = host.generate_packing(shape, c["rmin"], c["rmax"],
                                       c["porosity"], seed, device=_device())
    fluid = np.ones(shape, np.uint8)
    number = np.zeros(shape, np.int64)
    for i, (x, y, z, r) in enumerate(spheres.tolist()):
        host.place_sphere(fluid, x, y, z, r, number, i + 1)
    noise = torch.from_numpy(np.random.default_rng(seed).standard_normal(
        tuple(-(-n // 8) + 1 for n in shape), np.float32))
    smooth = torch.nn.functional.interpolate(
        noise[None, None], size=shape, mode="trilinear", align_corners=True)
    rho = (0.35 + 0.3 * torch.tanh(3 * smooth[0, 0])).numpy()
    return rho, fluid, number, len(spheres)


def prepare(case, seed):
    c = case
    if c["kind"] == "clusters":
        return dict(case=c, args=_two_phase(c, seed))
    doms = _domains(c, seed)
    if c["kind"] == "batch":
        b = batch.Batch(storage=STORAGE[c["storage"]])
        ids = [b.add(fluid, rho, params) for _, fluid, rho, params in doms]
        return dict(case=c, batch=b, lats=[b.lattice(i) for i in ids],
                    rho=_field_tensors(c, [d[0] for d in doms]))
    shape, fluid, rho, params = doms[0]
    if c["kind"] == "job":
        return dict(case=c, inputs=doms[0])
    lat = _lattice(c, shape, fluid, rho, params)
    if c["kind"] == "stats":
        lat.iterate(0, 1)
        return dict(case=c, lat=lat)
    s = dict(case=c, lat=lat, step=0, rho=_field_tensors(c, [shape])[0])
    if c["velocity"]:
        s["velocity"] = _field_tensors(c, [shape + (3,)])[0]
    return s


# ---- one pass ---------------------------------------------------------------

def _take(lat, field, out):
    kind = capi.DTYPE_F64 if out.dtype == torch.float64 else capi.DTYPE_F32
    capi.check(capi.lib().mlbm_download_field_device(
        lat.h, ctypes.c_int32(field), ctypes.c_int32(kind),
        ctypes.c_void_p(out.data_ptr())))
    return out


def run(state):
    c = state["case"]
    if c["kind"] == "clusters":
        rho, fluid, number, count = state["args"]
        row, liquid, gas = driver.cluster_stats(rho, fluid, number, RHO_L, RHO_G,
                                                count, device=0)
        return [row, liquid, gas]
    if c["kind"] == "stats":
        profile = state["lat"].plane_profile()
        return [state["lat"].stats(), *profile]
    if c["kind"] == "batch":
        state["batch"].iterate(c["steps"])
        return [_take(lat, capi.FIELD_RHO, out)
                for lat, out in zip(state["lats"], state["rho"])]
    if c["kind"] == "job":
        lat = _lattice(c, *state["inputs"])
        lat.iterate(0, c["steps"])
        rho = lat.field("rho", f64=c["storage"] == "f64")
        lat.close()
        return [rho]
    lat = state["lat"]
    lat.iterate(state["step"], c["steps"], write_velocity=c["velocity"])
    state["step"] += c["steps"]
    out = [_take(lat, capi.FIELD_RHO, state["rho"])]
    if c["velocity"]:
        out.append(_take(lat, capi.FIELD_VELOCITY, state["velocity"]))
    return out


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """A step reads and writes the state of every fluid node once: its 19
    populations, or, at tau = 1, where the collision leaves the equilibrium of
    the node's density and velocity, those 4 numbers.  Fields taken off are
    written once."""
    c = case
    real = 8 if c["storage"] == "f64" else 4
    pop = {"f32": 4, "f16": 2, "f64": 8}[c["storage"]]
    if c["kind"] == "batch":
        rng = np.random.default_rng(c["ny"])
        edges = np.arange(32, c["nx"] + 1, 16)
        nodes = fluid = 0.0
        for _ in range(c["ny"]):
            n = float(np.prod(rng.choice(edges, 3)))
            nodes += n
            fluid += n * float(rng.uniform(0.35, 0.65))
            rng.uniform(-2.0, 0.0)
    else:
        nodes = float(c["nx"] * c["ny"] * c["nz"])
        fluid = nodes * c["porosity"]
    if c["kind"] == "stats":
        return {"bytes": fluid * real + nodes / 8, "flops": fluid * 40}
    if c["kind"] == "clusters":
        return {"bytes": nodes * (4 + 1 + 8 + 16), "flops": nodes * 20}
    state = min(19 * pop, 4 * real) if c["tau"] == 1.0 else 19 * pop
    total = c["steps"] * (2 * state * fluid + nodes / 8)
    total += nodes * real * (4 if c["velocity"] else 1)
    if c["kind"] == "job":
        total += nodes * 5
    return {"bytes": total, "flops": 330.0 * fluid * c["steps"]}


# ---- the same in 64 bits -------------------------------------------------------

_EX = [0, -1, 0, 0, -1, -1, -1, -1, 0, 0]
_EY = [0, 0, -1, 0, -1, 1, 0, 0, -1, -1]
_EZ = [0, 0, 0, -1, 0, 0, -1, 1, -1, 1]
_E = [(_EX[i], _EY[i], _EZ[i]) for i in range(10)]
_E += [(-x, -y, -z) for x, y, z in _E[1:]]
_W = [1 / 3 if i == 0 else 1 / 18 if i in (1, 2, 3, 10, 11, 12) else 1 / 36
      for i in range(19)]
_OPP = [0] + [i + 9 if i < 10 else i - 9 for i in range(1, 19)]


def _pressure(p, rho):
    if p.carn_star:
        eta = rho
        return (rho * (p.T_Tc * 0.0943) * (1 + eta + eta**2 - eta**3)
                / (1 - eta) ** 3 - rho**2)
    return rho / 3 + p.G / 6 * (1 - torch.exp(-rho)) ** 2


def _psi(p, rho):
    if p.carn_star:
        return torch.sqrt(2 * (_pressure(p, rho) - rho / 3) / (p.G / 3))
    return 1 - torch.exp(-rho)


def _shifted(v, e, sign=1):
    s = tuple(sign * k for k in e)
    return v if s == (0, 0, 0) else torch.roll(v, s, (0, 1, 2))


def _evolve(shape, fluid, rho, p, steps):
    """Density and velocity after `steps`: pull streaming with halfway
    bounce-back, Shan-Chen force from the step's densities, velocity shift,
    BGK; slab nodes hold their density and the rest equilibrium."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    fl = torch.from_numpy(fluid).to(dev).bool()
    d0 = torch.from_numpy(rho).to(dev).double()
    solid = torch.full((), float(p.rhos), dtype=torch.float64, device=dev)
    x = torch.arange(shape[0], device=dev)[:, None, None]
    y = torch.arange(shape[1], device=dev)[None, :, None]
    inlet = x < p.inlet_width
    outlet = x >= shape[0] - p.outlet_width
    post = [w * d0 for w in _W]
    d = d0
    u = [torch.zeros_like(d0) for _ in range(3)]
    open_ = [_shifted(fl, e) for e in _E]  # the node a population comes from
    omega = 1.0 / float(p.tau)
    for s in range(steps):
        f = [torch.where(open_[i], _shifted(post[i], e), post[_OPP[i]])
             for i, e in enumerate(_E)]
        d = sum(f)
        if p.rho_inject_period and s % p.rho_inject_period == 0:
            d = torch.where(y < p.inject_position * shape[1],
                            d + float(p.rho_increment), d)
        d = torch.where(inlet, float(p.rho_inlet),
                        torch.where(outlet, float(p.rho_outlet), d))
        psi = _psi(p, torch.where(fl, d, solid))
        force, u = [0.0, 0.0, 0.0], [0.0, 0.0, 0.0]
        for i in range(1, 19):
            t = _W[i] * _shifted(psi, _E[i], -1)
            for a in range(3):
                if _E[i][a]:
                    force[a] = force[a] + _E[i][a] * t
                    u[a] = u[a] + _E[i][a] * f[i]
        held = (inlet | outlet)
        for a in range(3):
            u[a] = (u[a] - float(p.tau) * float(p.G) * psi * force[a]) / d
            u[a] = torch.where(held, 0.0, u[a])
        square = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        for i, e in enumerate(_E):
            eu = sum(e[a] * u[a] for a in range(3) if e[a]) if i else 0.0
            eq = _W[i] * d * (1 + 3 * eu + 4.5 * eu * eu - square)
            post[i] = torch.where(held, _W[i] * d, f[i] + (eq - f[i]) * omega)
        del f
    return (torch.where(fl, d, solid),
            torch.stack([torch.where(fl, v, 0.0) for v in u], -1))


def exact(case, seed):
    c = case
    if c["kind"] in ("clusters", "stats"):
        # counts, labels and sums over a field of the case's own precision
        return None
    out = []
    for shape, fluid, rho, p in _domains(c, seed):
        d, u = _evolve(shape, fluid, rho, p, c["steps"])
        out.append(d.cpu().numpy() if c["kind"] == "job" else d)
        if c["velocity"]:
            out.append(u)
    return out
