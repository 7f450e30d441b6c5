"""Workloads of the engine for timing and for comparing two builds of it.

Every case is one piece of a user's program over the public entry points (``FdmBackend``,
``FdmBatch``, ``rk4_final_state``): a block of integrator steps followed by reading the
state, a field evaluation of an uploaded state, a block of a parameter sweep, one
gradient.  ``prepare`` builds the problem (seeded inputs and the handle a program keeps),
``run`` advances it by one block and returns the state and the energies, ``work`` states
the compulsory bytes and operations, and ``exact`` gives the same results from plain
PyTorch in FP64.

A case is a dict of plain values:
  kind        steps | adaptive | field | sweep | adjoint
  nx, ny, nz  cells
  integrator  heun | rk4 | abm3 | dp45 | rk23
  terms       plain | uniaxial | cubic | dmi_sot
  precision   single | double
  mask        none | disk         (active cells: an ellipse in the x-y plane)
  periodic    none | x | xy       (10 demag images on each side)
  steps       steps in one pass (adaptive: the interval holds that many of the largest steps)
  loop        steps: True = one call per step, with statistics each time; False = one call
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from fullmag_gb300 import FdmBackend, FdmBatch, _abi
from fullmag_gb300.adjoint import rk4_final_state

MU0 = 4.0e-7 * math.pi
GAMMA = 2.211e5
HBAR, E_CHARGE = 1.054571817e-34, 1.602176634e-19

INTEGRATORS = {"heun": _abi.INTEGRATOR_HEUN, "rk4": _abi.INTEGRATOR_RK4, "abm3": _abi.INTEGRATOR_ABM3,
               "dp45": _abi.INTEGRATOR_DP45, "rk23": _abi.INTEGRATOR_RK23}
# field evaluations of one step
EVALUATIONS = {"heun": 2, "rk4": 4, "abm3": 2, "dp45": 6, "rk23": 3}

# materials with the term set they are used with: the plain permalloy-like film, a film with
# in-plane uniaxial anisotropy, an iron-like cubic volume, a perpendicular film with
# interfacial DMI driven by spin-orbit torque
MATERIALS = {
    "plain": dict(ms=8e5, a_ex=1.3e-11, alpha=0.05, d=(4e-9, 4e-9, 4e-9), b=(10e-3, 5e-3, 0.0)),
    "uniaxial": dict(ms=8e5, a_ex=1.3e-11, alpha=0.02, d=(3.90625e-9, 3.90625e-9, 3e-9), b=(-24.6e-3, 4.3e-3, 0.0),
                     ku1=5e3, u_axis=(1.0, 0.0, 0.0)),
    "cubic": dict(ms=1.4e6, a_ex=2.1e-11, alpha=0.01, d=(2e-9, 2e-9, 2e-9), b=None, kc1=-4.8e4),
    "dmi_sot": dict(ms=5.8e5, a_ex=1.5e-11, alpha=0.1, d=(2e-9, 2e-9, 1e-9), b=(0.0, 0.0, 20e-3), ku1=8e5,
                    u_axis=(0.0, 0.0, 1.0), dmi_d_interfacial=3e-3, sot_je=2e11, sot_xi_dl=0.15, sot_xi_fl=0.02,
                    sot_sigma=(0.0, 1.0, 0.0), sot_thickness=1e-9),
}


def _case(name, kind, nx, ny, nz, integrator="rk4", terms="plain", precision="single", mask="none", periodic="none",
          steps=1, loop=False):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, integrator=integrator, terms=terms, precision=precision, mask=mask,
             periodic=periodic, steps=steps, loop=loop)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest problem of the benchmark set: a box stepped one call at a time with its
        # energies after every step, the way an interactive runner drives it
        _case("box_64x32x4_heun", "steps", 64, 32, 4, "heun", steps=16, loop=True),
        # fixed-step film dynamics sampled every 50 steps
        _case("film_256x64_rk4", "steps", 256, 64, 1, "rk4", steps=50),
        # adaptive thin-film dynamics: a runner's loop over suggested steps to an output time
        _case("film_512x128_dp45", "adaptive", 512, 128, 1, "dp45", terms="uniaxial", steps=16),
        # the large volume
        _case("volume_256x256x64_rk4", "steps", 256, 256, 64, "rk4", terms="cubic", steps=6),
        # a patterned element: a disk in a box whose extents are no powers of two
        _case("disk_150x150x10_rk4", "steps", 150, 150, 10, "rk4", terms="plain", mask="disk", steps=20),
        # an extended film, periodic in the plane
        _case("film_256x256_periodic_rk4", "steps", 256, 256, 1, "rk4", periodic="xy", steps=20),
        # a skyrmion track: perpendicular film with DMI under a current
        _case("track_400x100_dmi_sot_rk4", "steps", 400, 100, 1, "rk4", terms="dmi_sot", steps=20),
        # the field and the energies of a state that the host holds (previews, hysteresis points,
        # host-side minimisers)
        _case("field_160x120x12", "field", 160, 120, 12, terms="cubic"),
        # double-precision state: film and volume
        _case("film_200x100_double_heun", "steps", 200, 100, 1, "heun", precision="double", steps=10, loop=True),
        _case("volume_128x128x16_double_rk4", "steps", 128, 128, 16, "rk4", terms="cubic", precision="double", steps=4,
              loop=True),
        # a block of a parameter sweep: films of uneven sizes and step limits in one batch
        # (nx, ny, nz are the largest extents, steps the most steps of a film)
        _case("sweep_24_films_dp45", "sweep", 256, 128, 4, "dp45", steps=64),
        # inverse design: the gradient with respect to the field map and the initial state
        _case("adjoint_256x64_rk4", "adjoint", 256, 64, 1, "rk4", steps=200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["box", "film", "adaptive", "volume", "disk", "periodic", "track", "field", "double_film",
                         "double_volume", "sweep", "adjoint"])
    terms = rng.choice(["plain", "uniaxial", "cubic"])
    fixed = rng.choice(["heun", "rk4", "rk4", "abm3"])
    if family == "box":
        return _case(None, "steps", _log_int(rng, 8, 96), _log_int(rng, 8, 64), rng.randint(2, 12), fixed, terms,
                     steps=rng.randint(8, 24), loop=True)
    if family == "film":
        return _case(None, "steps", _log_int(rng, 32, 1024), _log_int(rng, 16, 512), 1, fixed, terms,
                     steps=rng.randint(10, 50))
    if family == "adaptive":
        return _case(None, "adaptive", _log_int(rng, 32, 640), _log_int(rng, 16, 256), rng.choice([1, 1, 2, 5]),
                     rng.choice(["dp45", "dp45", "rk23"]), terms, steps=rng.randint(8, 20))
    if family == "volume":
        return _case(None, "steps", _log_int(rng, 40, 256), _log_int(rng, 40, 256), _log_int(rng, 12, 64), "rk4",
                     terms, steps=rng.randint(2, 6))
    if family == "disk":
        a = _log_int(rng, 48, 300)
        return _case(None, "steps", a, max(16, a - rng.randint(0, 12)), rng.randint(1, 12), fixed, terms, mask="disk",
                     steps=rng.randint(8, 20))
    if family == "periodic":
        return _case(None, "steps", 2 * _log_int(rng, 16, 256), _log_int(rng, 32, 512), rng.choice([1, 1, 4]), "rk4",
                     terms, periodic=rng.choice(["x", "xy"]), steps=rng.randint(8, 20))
    if family == "track":
        return _case(None, "steps", _log_int(rng, 96, 1024), _log_int(rng, 32, 200), rng.choice([1, 1, 2]), "rk4",
                     "dmi_sot", steps=rng.randint(8, 20))
    if family == "field":
        return _case(None, "field", _log_int(rng, 16, 256), _log_int(rng, 16, 256), _log_int(rng, 1, 24), terms=terms)
    if family == "double_film":
        return _case(None, "steps", _log_int(rng, 32, 512), _log_int(rng, 16, 256), 1, fixed, terms,
                     precision="double", steps=rng.randint(4, 10), loop=True)
    if family == "double_volume":
        return _case(None, "steps", _log_int(rng, 24, 160), _log_int(rng, 24, 128), _log_int(rng, 4, 24), "rk4", terms,
                     precision="double", steps=rng.randint(2, 4), loop=True)
    if family == "sweep":
        return _case(None, "sweep", _log_int(rng, 48, 256), _log_int(rng, 32, 128), rng.choice([1, 2, 4]), "dp45",
                     steps=rng.randint(24, 64))
    return _case(None, "adjoint", _log_int(rng, 32, 256), _log_int(rng, 16, 96), 1, "rk4", steps=rng.randint(50, 200))


# ---- inputs ----

SWEEP_FILMS = 24


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _unit(v):
    return v / v.norm(dim=0, keepdim=True)


def _smooth_state(nx, ny, nz, terms, g):
    """Seeded unit vectors (3, nz, ny, nx), FP64: random directions smoothed by three passes of
    a 6-neighbour box filter (domains a few cells wide); the driven film starts from +x and
    the perpendicular film from +z, each with a smoothed random tilt."""
    v = torch.randn(3, nz, ny, nx, device="cuda", dtype=torch.float64, generator=g)
    for _ in range(3):
        acc = v.clone()
        for ax, ext in ((1, nz), (2, ny), (3, nx)):
            if ext > 1:
                acc = acc + v.roll(1, ax) + v.roll(-1, ax)
        v = acc / 7.0
    if terms in ("uniaxial", "dmi_sot"):
        v = 0.2 * v / v.norm(dim=0).mean()
        if terms == "uniaxial":
            v[0] += 1.0
        else:
            a = 2.0 * math.pi / 48.0 * torch.arange(nx, device="cuda", dtype=torch.float64)
            v[0] += a.sin()
            v[2] += a.cos()
    return _unit(v)


def _mask(case):
    """The ellipse that fills the box in the plane, (nz, ny, nx) bool, or None."""
    if case["mask"] == "none":
        return None
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x = (torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5) / nx * 2.0 - 1.0
    y = (torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5) / ny * 2.0 - 1.0
    return (y[:, None] ** 2 + x[None, :] ** 2 <= 1.0).expand(nz, ny, nx).contiguous()


def _aos(v):
    return np.ascontiguousarray(v.reshape(3, -1).t().cpu().numpy())


def _dt(case):
    """Step size: well inside the stability limit of the exchange modes of the material."""
    return {"plain": 5e-14, "uniaxial": 5e-14, "cubic": 2e-14, "dmi_sot": 2e-14}[case["terms"]]


def _spec(case, seed):
    """One problem: plan keywords without the state, the FP64 state and the mask."""
    mat = MATERIALS[case["terms"]]
    kw = {k: v for k, v in mat.items() if k not in ("d", "b")}
    dx, dy, dz = mat["d"]
    kw.update(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=dx, dy=dy, dz=dz, gamma=GAMMA)
    if mat["b"] is not None:
        kw["h_ext"] = tuple(b / MU0 for b in mat["b"])
    mask = _mask(case)
    m = _smooth_state(case["nx"], case["ny"], case["nz"], case["terms"], _generator(seed))
    if mask is not None:
        m = m * mask
    return kw, m, mask


def _sweep_spec(case, seed, states=True):
    """Films with extents up to the case's, material and in-plane field drawn from the seed's
    generator, and a largest step per film that divides the pass's interval:
    [(plan keywords, FP64 state or None, largest step)]."""
    r = np.random.default_rng(int(seed) & 0x7FFFFFFF)
    shapes = np.random.default_rng(1000 * case["nx"] + case["ny"])  # the same sizes for every seed
    films = []
    for _ in range(SWEEP_FILMS):
        nx = int(shapes.integers(16, case["nx"] + 1))
        ny = int(shapes.integers(16, case["ny"] + 1))
        nz = int(shapes.choice([z for z in (1, 2, 4) if z <= case["nz"]]))
        k = int(shapes.integers(max(4, case["steps"] // 2), case["steps"] + 1))
        b, ang = r.uniform(0.0, 0.1), r.uniform(0.0, 2.0 * math.pi)
        kw = dict(nx=nx, ny=ny, nz=nz, dx=4e-9, dy=4e-9, dz=4e-9, ms=r.uniform(4e5, 1.2e6),
                  a_ex=r.uniform(5e-12, 2e-11), alpha=r.uniform(0.005, 0.1), gamma=GAMMA,
                  h_ext=(b * math.cos(ang) / MU0, b * math.sin(ang) / MU0, 0.0))
        state_seed = r.integers(1 << 30)
        m = _smooth_state(nx, ny, nz, "plain", _generator(state_seed)) if states else None
        films.append((kw, m, _interval(case) / k))
    return films


def _interval(case):
    """Simulated time of an adaptive pass."""
    return case["steps"] * (4e-14 if case["kind"] == "sweep" else _dt(case))


def _field_map(case, seed):
    """The trainable in-plane map (n, 2), N(0, 2 mT), and the target pattern (n, 3)."""
    g = _generator(seed + 7)
    n = case["nx"] * case["ny"]
    b = (2e-3 * torch.randn(n, 2, device="cuda", dtype=torch.float64, generator=g)).float()
    t = _smooth_state(case["nx"], case["ny"], 1, "uniaxial", g)
    return b, t.reshape(3, -1).t().contiguous().float()


_PERIODIC = {"none": (0, 0, 0), "x": (1, 0, 0), "xy": (1, 1, 0)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        films = _sweep_spec(case, seed)
        batch = FdmBatch([dict(kw, m0=_aos(m), integrator=_abi.INTEGRATOR_DP45, adaptive_max_error=1e-5,
                               adaptive_dt_max=cap) for kw, m, cap in films])
        return dict(kind=kind, batch=batch, interval=_interval(case), dt0=max(cap for _, _, cap in films), t=0.0)
    kw, m, mask = _spec(case, seed)
    plan = dict(kw, m0=_aos(m), integrator=INTEGRATORS[case["integrator"]],
                precision=_abi.PRECISION_DOUBLE if case["precision"] == "double" else _abi.PRECISION_SINGLE)
    if mask is not None:
        plan["active_mask"] = mask.to(torch.uint8).cpu().numpy()
    if case["integrator"] in ("dp45", "rk23"):
        plan.update(adaptive_max_error=1e-5, adaptive_dt_max=_dt(case))
    if case["periodic"] != "none":
        plan.update(periodic=_PERIODIC[case["periodic"]])
    be = FdmBackend(**plan)
    s = dict(kind=kind, be=be, dt=_dt(case), steps=case["steps"], loop=case["loop"], t=0.0,
             single=case["precision"] == "single")
    if kind == "adaptive":
        s["interval"] = _interval(case)
    if kind == "field":
        s["m"] = plan["m0"]
    if kind == "adjoint":
        b, target = _field_map(case, seed)
        s["m0"] = torch.from_numpy(plan["m0"]).float().requires_grad_()
        s["b"] = b.cpu().requires_grad_()
        s["target"] = target.cpu()
    return s


# ---- one pass ----

class _DeviceView:
    """A component of the engine's device-resident state as a CUDA array."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3)


def _device_m(be):
    p = [ctypes.c_void_p() for _ in range(3)]
    be._check(be.lib.fullmag_fdm_backend_device_magnetization(be.handle, *[ctypes.byref(q) for q in p]),
              "device_magnetization")
    return [torch.as_tensor(_DeviceView(be, q.value, be.n), device="cuda") for q in p]


STATS = ("exchange_energy_joules", "demag_energy_joules", "external_energy_joules", "anisotropy_energy_joules",
         "cubic_energy_joules", "dmi_energy_joules", "total_energy_joules", "max_effective_field_amplitude",
         "max_demag_field_amplitude", "max_rhs_amplitude")


def _stats(st, single):
    """Energies and norms in the precision of the state they are sums over."""
    t = np.float32 if single else np.float64
    return {k: t(st[k]) for k in STATS}


def run(state):
    kind = state["kind"]
    if kind == "sweep":
        state["t"] += state["interval"]
        batch = state["batch"]
        batch.step_until(state["t"], state["dt0"])
        return {"m": [batch.copy_field(i).astype(np.float32) for i in range(len(batch))]}
    be = state["be"]
    if kind == "field":
        be.upload(state["m"])
        be.refresh()
        st = be.stats()
        return {"h_eff": be.copy_field(_abi.OBSERVABLE_H_EFF, np.float32),
                "h_demag": be.copy_field(_abi.OBSERVABLE_H_DEMAG, np.float32), **_stats(st, True)}
    if kind == "adjoint":
        state["m0"].grad = state["b"].grad = None
        m = rk4_final_state(state["m0"], state["b"], be, state["dt"], state["steps"])
        loss = (m - state["target"]).square().mean()
        loss.backward()
        return {"m": m.detach(), "grad_b": state["b"].grad, "grad_m0": state["m0"].grad}
    if kind == "adaptive":
        end = state["t"] + state["interval"]
        dt = state["dt"]
        while state["t"] < end * (1.0 - 1e-12):
            st = be.step(min(dt, end - state["t"]))
            state["t"], dt = st["time_seconds"], st["suggested_next_dt"]
    elif state["loop"]:
        for _ in range(state["steps"]):
            st = be.step(state["dt"])
    else:
        st = be.step_many(state["dt"], state["steps"])
    return {"m": _device_m(be) if state["single"] else be.copy_field(_abi.OBSERVABLE_M),
            **_stats(st, state["single"])}


# ---- compulsory work ----

def _grid_work(nx, ny, nz, precision, periodic="none"):
    """(bytes, operations) of one field evaluation, each of which needs the whole state that the
    last one gave: the state read and one vector field written, the demag tensor's unique
    spectrum read; six half-complex transforms of the padded grid, the tensor product, the
    stencil and the local terms."""
    w = 8 if precision == "double" else 4
    n = nx * ny * nz
    per = _PERIODIC[periodic]
    p = [nx if per[0] else 2 * nx, ny if per[1] else 2 * ny, 1 if nz == 1 else 2 * nz]
    cells = p[0] * p[1] * p[2]
    comps = 4 if nz == 1 else 6
    unique = [(q if f else q // 2 + 1) for q, f in zip(p, per)]
    unique[0] = p[0] // 2 + 1
    tensor = comps * unique[0] * unique[1] * unique[2] * (2 if any(per) else 1)
    # zero planes make the x and y passes cheaper than a full transform: x lines of real rows
    # only, y lines of the rows' spectra, z lines of everything
    lg = [math.log2(q) if q > 1 else 0.0 for q in p]
    fft = 2.5 * (ny * nz * p[0] * lg[0] + nz * p[0] * p[1] * lg[1] + cells * lg[2])
    return 6 * w * n + tensor * w, 6 * fft + 15 * cells + 90 * n


def work(case):
    if case["kind"] == "sweep":
        by = fl = 0.0
        for kw, _, cap in _sweep_spec(case, 0, states=False):
            b, f = _grid_work(kw["nx"], kw["ny"], kw["nz"], "single")
            evals = EVALUATIONS["dp45"] * round(_interval(case) / cap)
            by, fl = by + b * evals, fl + f * evals
        return {"bytes": by, "flops": fl}
    b, f = _grid_work(case["nx"], case["ny"], case["nz"], case["precision"], case["periodic"])
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "field":
        return {"bytes": b + (24 + 2 * 12) * n, "flops": f}
    evals = EVALUATIONS[case["integrator"]] * case["steps"]
    if case["kind"] == "adjoint":
        evals *= 3  # forward, recomputed forward, reverse
    return {"bytes": b * evals, "flops": f * evals}


# ---- the same results in FP64 ----

ASYMPTOTIC = 40  # cells: beyond, the tensor is the point dipole's


def _newell_f(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    r = torch.sqrt(x2 + y2 + z2)
    acc = (2.0 * x2 - y2 - z2) * r / 6.0

    def log_term(q, s):
        t = torch.where(s > 1e-300, 2.0 * q * (q + r) / s.clamp_min(1e-300), torch.zeros_like(s))
        return torch.where(t > -1.0, torch.log1p(t.clamp_min(-1.0 + 1e-16)), torch.zeros_like(t))

    acc = acc + y * (z2 - x2) / 4.0 * log_term(y, x2 + z2) + z * (y2 - x2) / 4.0 * log_term(z, x2 + y2)
    at = torch.where(x.abs() > 1e-300, torch.atan(y * z / torch.where(x.abs() > 1e-300, x * r, torch.ones_like(x))),
                     torch.zeros_like(x))
    return acc - x * y * z * at


def _newell_g(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    r = torch.sqrt(x2 + y2 + z2)
    acc = -x * y * r / 3.0

    def log_term(q, s):
        t = torch.where(s > 1e-300, 2.0 * q * (q + r) / s.clamp_min(1e-300), torch.zeros_like(s))
        return torch.where(t > -1.0, torch.log1p(t.clamp_min(-1.0 + 1e-16)), torch.zeros_like(t))

    def atan(num, q):
        ok = q.abs() > 1e-300
        return torch.where(ok, torch.atan(num / torch.where(ok, q * r, torch.ones_like(q))), torch.zeros_like(q))

    acc = acc + x * y * z * log_term(z, x2 + y2) / 2.0 + y * (3.0 * z2 - y2) * log_term(x, y2 + z2) / 12.0 \
        + x * (3.0 * z2 - x2) * log_term(y, x2 + z2) / 12.0
    return acc - z2 * z / 6.0 * atan(x * y, z) - y2 * z / 2.0 * atan(x * z, y) - x2 * z / 2.0 * atan(y * z, x)


class _Tensor:
    """The Newell tensor at whole-cell offsets: the 27-point second difference of f and g inside
    the asymptotic distance (compensated sums), the point dipole beyond."""

    def __init__(self, d, reach):
        self.d, self.v = d, d[0] * d[1] * d[2]
        ext = [min(r, ASYMPTOTIC) + 2 for r in reach]
        z, y, x = torch.meshgrid(*[(torch.arange(e, device="cuda", dtype=torch.float64) - 1.0) * h
                                   for e, h in zip(ext[::-1], d[::-1])], indexing="ij")
        origin = (x == 0) & (y == 0) & (z == 0)
        tabs = [_newell_f(x, y, z), _newell_f(y, x, z), _newell_f(z, y, x),
                _newell_g(x, y, z), _newell_g(x, z, y), _newell_g(y, z, x)]
        near = []
        for t in tabs:
            t = torch.where(origin, torch.zeros_like(t), t)
            s = torch.zeros([e - 2 for e in ext[::-1]], device="cuda", dtype=torch.float64)
            c = torch.zeros_like(s)
            for dc in range(3):
                for db in range(3):
                    for da in range(3):
                        w = 1.0
                        for q in (da, db, dc):
                            w *= 2.0 if q == 1 else -1.0
                        v = w * t[dc:dc + s.shape[0], db:db + s.shape[1], da:da + s.shape[2]]
                        u = s + v
                        c = c + torch.where(s.abs() >= v.abs(), (s - u) + v, (v - u) + s)
                        s = u
            near.append((s + c) / (4.0 * math.pi * self.v))
        self.near = torch.stack(near)

    def at(self, i, j, k):
        """(6, len(k), len(j), len(i)) at signed offsets: xx yy zz xy xz yz."""
        k3, j3, i3 = torch.meshgrid(k, j, i, indexing="ij")
        a = [q.abs() for q in (i3, j3, k3)]
        far = (a[0] >= ASYMPTOTIC) | (a[1] >= ASYMPTOTIC) | (a[2] >= ASYMPTOTIC) | \
            (a[0] ** 2 + a[1] ** 2 + a[2] ** 2 >= ASYMPTOTIC ** 2)
        idx = [q.clamp_max(s - 1) for q, s in zip(a[::-1], self.near.shape[1:])]
        out = self.near[:, idx[0], idx[1], idx[2]]
        x, y, z = (q.double() * h for q, h in zip(a, self.d))
        r2 = (x * x + y * y + z * z).clamp_min(1e-60)
        r = torch.sqrt(r2)
        s3, s5 = self.v / (4.0 * math.pi * r2 * r), -3.0 * self.v / (4.0 * math.pi * r2 * r2 * r)
        dip = torch.stack([s3 + s5 * x * x, s3 + s5 * y * y, s3 + s5 * z * z, s5 * x * y, s5 * x * z, s5 * y * z])
        out = torch.where(far, dip, out)
        sg = [torch.where(q < 0, -1.0, 1.0).double() for q in (i3, j3, k3)]
        out[3] *= sg[0] * sg[1]
        out[4] *= sg[0] * sg[2]
        out[5] *= sg[1] * sg[2]
        return out


class _Exact:
    """Fields, energies and right-hand side of one problem in FP64 on (3, nz, ny, nx) tensors."""

    def __init__(self, kw, mask=None, periodic=(0, 0, 0), images=10):
        self.kw, self.mask, self.per = kw, mask, periodic
        self.n3 = (kw["nz"], kw["ny"], kw["nx"])
        self.d = (kw["dx"], kw["dy"], kw["dz"])
        n = (kw["nx"], kw["ny"], kw["nz"])
        p = [q if f else 2 * q for q, f in zip(n, periodic)]
        if n[2] == 1 and not periodic[2]:
            p[2] = 1
        im = [images if f else 0 for f in periodic]
        tensor = _Tensor(self.d, [q * (1 + 2 * g) for q, g in zip(n, im)])
        ax = []
        for a in range(3):
            i = torch.arange(p[a], device="cuda")
            ax.append(i if periodic[a] or p[a] == 1 else torch.where(i < n[a], i, i - p[a]))
        live = torch.ones(p[::-1], device="cuda", dtype=torch.float64)
        for a in range(3):
            if not periodic[a] and p[a] > 1:
                live.select(2 - a, n[a]).zero_()
        acc = torch.zeros([6] + p[::-1], device="cuda", dtype=torch.float64)
        for mz in range(-im[2], im[2] + 1):
            for my in range(-im[1], im[1] + 1):
                for mx in range(-im[0], im[0] + 1):
                    acc += tensor.at(ax[0] + mx * n[0], ax[1] + my * n[1], ax[2] + mz * n[2])
        acc *= live * kw["ms"]
        self.p = p[::-1]
        self.spec = torch.fft.rfftn(acc, dim=(1, 2, 3))
        if not any(periodic):
            self.spec = self.spec.real.contiguous()

    def shifted(self, m, a, s):
        """m at the neighbour s = +-1 along axis a (0 x): the cell itself where there is none."""
        dim = 3 - a
        out = m.roll(-s, dim)
        edge = self.n3[2 - a] - 1 if s > 0 else 0
        own = torch.zeros(self.n3, device="cuda", dtype=torch.bool)
        if not self.per[a]:
            own.select(dim - 1, edge).fill_(True)
        if self.mask is not None:
            own = own | ~self.mask.roll(-s, dim - 1)
        return torch.where(own, m, out) if bool(own.any()) else out

    def fields(self, m):
        kw = self.kw
        h_ex = torch.zeros_like(m)
        nb = {}
        for a in range(3):
            if self.n3[2 - a] > 1:
                nb[a] = (self.shifted(m, a, 1), self.shifted(m, a, -1))
                h_ex = h_ex + (nb[a][0] + nb[a][1] - 2.0 * m) / self.d[a] ** 2
        h_ex = h_ex * (2.0 * kw["a_ex"] / (MU0 * kw["ms"]))
        f = torch.fft.rfftn(m, s=self.p, dim=(1, 2, 3))
        xx, yy, zz, xy, xz, yz = self.spec
        h = torch.stack([xx * f[0] + xy * f[1] + xz * f[2], xy * f[0] + yy * f[1] + yz * f[2],
                         xz * f[0] + yz * f[1] + zz * f[2]])
        h_d = -torch.fft.irfftn(h, s=self.p, dim=(1, 2, 3))[:, :self.n3[0], :self.n3[1], :self.n3[2]]
        h = h_ex + h_d
        if "h_ext" in kw:
            h = h + torch.tensor(kw["h_ext"], device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
        if "ku1" in kw:
            u = torch.tensor(kw["u_axis"], device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
            h = h + 2.0 * kw["ku1"] / (MU0 * kw["ms"]) * (m * u).sum(0) * u
        if "kc1" in kw:
            s = m * m
            h = h - 2.0 * kw["kc1"] / (MU0 * kw["ms"]) * m * (s.sum(0) - s)
        if "dmi_d_interfacial" in kw:
            gx = (nb[0][0] - nb[0][1]) / (2.0 * self.d[0])
            gy = (nb[1][0] - nb[1][1]) / (2.0 * self.d[1])
            h = h + 2.0 * kw["dmi_d_interfacial"] / (MU0 * kw["ms"]) * torch.stack([gx[2], gy[2], -(gx[0] + gy[1])])
        if self.mask is not None:
            h, h_d, h_ex = h * self.mask, h_d * self.mask, h_ex * self.mask
        return h_d, h, nb

    def rhs_of(self, m, h):
        kw = self.kw
        p = torch.linalg.cross(m, h, dim=0)
        k = -kw["gamma"] / (1.0 + kw["alpha"] ** 2) * (p + kw["alpha"] * torch.linalg.cross(m, p, dim=0))
        if "sot_je" in kw:
            s = torch.tensor(kw["sot_sigma"], device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
            amp = abs(kw["sot_je"]) * HBAR / (2.0 * E_CHARGE * MU0 * kw["ms"] * kw["sot_thickness"])
            k = k + amp * (-kw["sot_xi_dl"] * ((m * s).sum(0) * m - s)
                           + kw["sot_xi_fl"] * torch.linalg.cross(m, s.expand_as(m), dim=0))
        return k

    def rhs(self, m, extra=None):
        h = self.fields(m)[1]
        return self.rhs_of(m, h if extra is None else h + extra)

    def normalised(self, v):
        if self.mask is None:
            return _unit(v)
        return v / torch.where(self.mask, v.norm(dim=0), torch.ones((), device="cuda", dtype=torch.float64))

    def stats(self, m):
        kw = self.kw
        vol = self.d[0] * self.d[1] * self.d[2]
        h_d, h, nb = self.fields(m)
        e = dict.fromkeys(STATS, 0.0)
        for a, (up, _) in nb.items():
            pair = (up - m) ** 2 if self.mask is None else (up - m) ** 2 * self.mask
            e["exchange_energy_joules"] += float(kw["a_ex"] * vol * pair.sum()) / self.d[a] ** 2
        e["demag_energy_joules"] = float(-0.5 * MU0 * kw["ms"] * vol * (m * h_d).sum())
        if "h_ext" in kw:
            hx = torch.tensor(kw["h_ext"], device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
            e["external_energy_joules"] = float(-MU0 * kw["ms"] * vol * (m * hx).sum())
        if "ku1" in kw:
            u = torch.tensor(kw["u_axis"], device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
            e["anisotropy_energy_joules"] = float(-vol * kw["ku1"] * ((m * u).sum(0) ** 2).sum())
        if "kc1" in kw:
            s = m * m
            e["cubic_energy_joules"] = float(vol * kw["kc1"] * (s[0] * s[1] + s[1] * s[2] + s[0] * s[2]).sum())
        if "dmi_d_interfacial" in kw:
            gx = (nb[0][0] - nb[0][1]) / (2.0 * self.d[0])
            gy = (nb[1][0] - nb[1][1]) / (2.0 * self.d[1])
            e["dmi_energy_joules"] = float(vol * kw["dmi_d_interfacial"] *
                                           (m[2] * (gx[0] + gy[1]) - m[0] * gx[2] - m[1] * gy[2]).sum())
        e["total_energy_joules"] = sum(e[k] for k in STATS[:6])
        e["max_effective_field_amplitude"] = float(h.norm(dim=0).max())
        e["max_demag_field_amplitude"] = float(h_d.norm(dim=0).max())
        e["max_rhs_amplitude"] = float(self.rhs_of(m, h).norm(dim=0).max())
        return {k: np.float64(v) for k, v in e.items()}

    def rk4(self, m, dt, extra=None):
        k1 = self.rhs(m, extra)
        k2 = self.rhs(self.normalised(m + 0.5 * dt * k1), extra)
        k3 = self.rhs(self.normalised(m + 0.5 * dt * k2), extra)
        k4 = self.rhs(self.normalised(m + dt * k3), extra)
        return self.normalised(m + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4))

    def heun(self, m, dt):
        k1 = self.rhs(m)
        k2 = self.rhs(self.normalised(m + dt * k1))
        return self.normalised(m + 0.5 * dt * (k1 + k2))

    def fixed(self, m, dt, steps, integrator):
        if integrator == "rk4":
            for _ in range(steps):
                m = self.rk4(m, dt)
        elif integrator == "heun":
            for _ in range(steps):
                m = self.heun(m, dt)
        else:  # three Heun steps, then the Adams-Bashforth predictor and the Adams-Moulton corrector
            hist = []
            for s in range(steps):
                if s < 3:
                    m = self.heun(m, dt)
                    f = self.rhs(m)
                else:
                    p = self.normalised(m + dt / 12.0 * (23.0 * hist[0] - 16.0 * hist[1] + 5.0 * hist[2]))
                    f = self.rhs(p)
                    m = self.normalised(m + dt / 12.0 * (5.0 * f + 8.0 * hist[0] - hist[1]))
                hist = [f] + hist[:2]
        return m

    TABLEAU = {
        "dp45": (((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
                  (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
                  (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
                  (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84)),
                 (71 / 57600, 0.0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40), 0.2),
        "rk23": (((1 / 2,), (0.0, 3 / 4), (2 / 9, 1 / 3, 4 / 9)), (-5 / 72, 1 / 12, 1 / 9, -1 / 8), 1 / 3),
    }

    def adaptive(self, m, t_end, dt0, dt_max, integrator, tol=1e-5, headroom=0.8):
        rows, err_w, order = self.TABLEAU[integrator]
        t, dt, k1 = 0.0, dt0, self.rhs(m)
        while t < t_end * (1.0 - 1e-12):
            dt = min(dt, t_end - t)
            k = [k1]
            for row in rows:
                y = self.normalised(m + dt * sum(c * q for c, q in zip(row, k) if c))
                k.append(self.rhs(y))
            err = float((dt * sum(c * q for c, q in zip(err_w, k) if c)).norm(dim=0).max())
            want = min(max(headroom * dt * (tol / err) ** order, 1e-18), dt_max) if err > 0.0 else dt_max
            if err <= tol:
                t, m, k1 = t + dt, y, k[-1]
            dt = want
        return m


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        out = []
        for kw, m, cap in _sweep_spec(case, seed):
            x = _Exact(kw)
            out.append(_aos(x.adaptive(m, _interval(case), cap, cap, "dp45")))
        return {"m": out}
    kw, m, mask = _spec(case, seed)
    x = _Exact(kw, mask, _PERIODIC[case["periodic"]])
    if kind == "field":
        h_d, h, _ = x.fields(m)
        return {"h_eff": _aos(h), "h_demag": _aos(h_d), **x.stats(m)}
    if kind == "adjoint":
        b, target = _field_map(case, seed)
        m0 = m.float().double().requires_grad_()
        bm = b.double().requires_grad_()
        hm = torch.nn.functional.pad(bm, (0, 1)).t().reshape(3, 1, case["ny"], case["nx"]) / MU0
        y = m0
        for _ in range(case["steps"]):
            y = x.rk4(y, _dt(case), hm)
        final = y.reshape(3, -1).t()
        (final - target.double()).square().mean().backward()
        return {"m": final.detach(), "grad_b": bm.grad, "grad_m0": m0.grad.reshape(3, -1).t().contiguous()}
    if kind == "adaptive":
        m = x.adaptive(m, _interval(case), _dt(case), _dt(case), case["integrator"])
    else:
        m = x.fixed(m, _dt(case), case["steps"], case["integrator"])
    e = x.stats(m)
    if "sot_je" in kw:  # the engine carries the torque in its field: this maximum includes it
        e["max_effective_field_amplitude"] = None
    return {"m": [q.reshape(-1) for q in m] if case["precision"] == "single" else _aos(m), **e}
