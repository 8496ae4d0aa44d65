"""Workloads of the coupled thermal lattice-Boltzmann step, timed through the public Python interface.

Each case is one pass of what a program that uses the library does between two looks at its
solution: advance a lattice (or many) by a number of time steps and read the fields and the
Nusselt / Reynolds numbers back.  Every run starts from a convecting state (a temperature
profile with seeded noise and a pair of rolls), loaded through the state-transfer calls, so that
velocities, temperatures and their lag state are those of a solution under way.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, "-2d-3d-_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import lbmgpu  # noqa: E402
from lbmgpu.abi import rb_params  # noqa: E402
from lbmgpu.server import StreamBatch  # noqa: E402

# numpy type of what a caller keeps of a field, by storage form
DTYPES = {"fp64": np.float64, "fp64x": np.float64, "fp32": np.float32, "fp16": np.float16}
# bytes of a stored population
ESIZE = {"fp64": 8, "fp64x": 8, "fp32": 4, "fp16": 2}
EXACT_CELL_STEPS = 2.0e9  # the 64-bit statement takes about 15 seconds for so many cell updates


def _solve(name, dim, nx, ny, nz, Ra, precision, steps, pattern="AB", U=0.1, Pr=0.71, kind="solve", periodic_x=None):
    return {"name": name, "kind": kind, "dim": dim, "nx": nx, "ny": ny, "nz": nz, "Ra": Ra, "Pr": Pr, "U": U,
            "precision": precision, "pattern": pattern, "steps": steps,
            "periodic_x": (dim == 2) if periodic_x is None else periodic_x}


def listed():
    return [
        # the smallest solve of the served stream at FP64 accuracy: one chunk of 500 steps between two Nu samples
        _solve("served_2d_128x64_fp64x", 2, 128, 64, 1, 1e5, "fp64x", 500),
        # the reference's own 2D case in the reference's arithmetic
        _solve("rb2d_256x128_fp64", 2, 256, 128, 1, 1e5, "fp64", 500),
        # a large 2D cell in FP32, walls on all sides, sizes off any power of two
        _solve("rb2d_2050x1025_fp32", 2, 2050, 1025, 1, 1e7, "fp32", 300, periodic_x=False),
        # a small cube in half storage (stochastic rounding), a chunk of a sweep over parameters
        _solve("rb3d_96_fp16", 3, 96, 96, 96, 1e6, "fp16", 400),
        # a box of odd, uneven sides in FP32, x periodic
        _solve("rb3d_161x97x131_fp32", 3, 161, 97, 131, 1e6, "fp32", 300, periodic_x=True),
        # the 128^3 cube in the reference's arithmetic
        _solve("rb3d_128_fp64", 3, 128, 128, 128, 1e7, "fp64", 40),
        # the 256^3 cube at FP64 accuracy, resident in HBM
        _solve("rb3d_256_fp64x", 3, 256, 256, 256, 1e7, "fp64x", 100),
        # the same as a whole job: every field in from host arrays, 200 steps, T and Nu/Re out
        _solve("job3d_256_fp64x", 3, 256, 256, 256, 1e7, "fp64x", 200, kind="job"),
        # the largest cube, half storage, in place
        _solve("rb3d_384_fp16_inplace", 3, 384, 384, 384, 1e9, "fp16", 128, pattern="AA", U=0.07),
        # many 2D instances of uneven sizes, Ra and Pr advanced together
        {"name": "batch_2d_fp32", "kind": "batch", "dim": 2, "members": 60, "ny_min": 64, "ny_max": 512,
         "precision": "fp32", "steps": 200, "spec_seed": 20261203},
        # a served mix of 2D and 3D solves at FP64 accuracy, one stream per solve
        {"name": "served_mix_fp64x", "kind": "streams", "dim": 0, "members": 12, "ny_min": 64, "ny_max": 160,
         "precision": "fp64x", "steps": 50, "spec_seed": 7},
        # the reference's subroutines called one by one from the caller's own loop
        _solve("stages3d_64_fp64", 3, 64, 64, 64, 1e6, "fp64", 20, kind="stages"),
    ]


def draw(rng):
    """One more case over the same ranges: storage forms, patterns, boundaries, sizes (odd ones among
    them) and kinds; the number of steps keeps a pass below about 0.3 s."""
    def edge(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return max(lo, min(hi, n + (n + 1) % 2 if rng.random() < 0.5 else n))

    kind = rng.choices(["solve", "job", "stages", "batch", "streams"], [14, 2, 1, 2, 1])[0]
    if kind in ("batch", "streams"):
        prec = rng.choice(["fp32", "fp16"]) if kind == "batch" else "fp64x"
        top = rng.choice([128, 256, 384] if kind == "batch" else [96, 128])
        return {"kind": kind, "dim": rng.choice([0, 2]), "members": rng.randint(4, 40 if kind == "batch" else 12),
                "ny_min": 48, "ny_max": top if kind == "streams" else min(top, 256), "precision": prec,
                "steps": rng.randint(20, 50), "spec_seed": rng.randrange(1 << 30)}
    dim = rng.choice([2, 3, 3])
    prec = "fp64" if kind == "stages" else rng.choice(["fp64", "fp64x", "fp64x", "fp32", "fp32", "fp16"])
    if dim == 2:
        ny = edge(48, 1400)
        nx, nz = int(ny * rng.uniform(0.8, 2.6)), 1
    else:
        ny = edge(24, 224)
        nx, nz = int(ny * rng.uniform(0.7, 1.5)), int(ny * rng.uniform(0.5, 1.3))
    cells = nx * ny * nz
    rate = {"fp64": 0.9e9, "fp64x": 8e9, "fp32": 14e9, "fp16": 14e9}[prec] * (3.0 if dim == 2 else 1.0)
    step_s = max(cells / rate, 2e-5) * (8 if kind == "stages" else 1)
    steps = max(4, min(500, int(rng.uniform(0.1, 0.25) / step_s)))
    c = _solve("", dim, nx, ny, nz, _stable_ra(rng.choice([1e5, 1e6, 1e7]), 0.71, 0.1, ny), prec, steps,
               pattern="AA" if kind == "solve" and prec != "fp64x" and rng.random() < 0.3 else "AB", kind=kind,
               periodic_x=rng.random() < 0.5)
    del c["name"]
    return c


def _stable_ra(Ra, Pr, U, L):
    """The Rayleigh number, lowered where the relaxation time would come closer to 1/2 than 0.02."""
    return min(Ra, 3.0 * Pr * (U * math.sqrt(3.0) * L / 0.02) ** 2)


def _member_cases(case):
    """The lattices of a batched or served case, uneven sizes drawn once from the case's own number."""
    rng = random.Random(case["spec_seed"])
    sizes = [n for n in (48, 64, 96, 128, 160, 192, 256, 384, 512) if case["ny_min"] <= n <= case["ny_max"]]
    out = []
    for m in range(case["members"]):
        dim = case["dim"] or (2 if m % 2 == 0 else 3)
        ny, Pr = rng.choice(sizes), rng.choice([0.71, 7.0])
        Ra = _stable_ra(math.exp(rng.uniform(math.log(1e4), math.log(1e8))), Pr, 0.1, ny)
        out.append(_solve("", dim, 2 * ny if dim == 2 else ny, ny, 1 if dim == 2 else ny, Ra, case["precision"],
                          case["steps"], Pr=Pr))
    return out


def _params(c, seed):
    return rb_params(dim=c["dim"], nx=c["nx"], ny=c["ny"], nz=c["nz"], Ra=c["Ra"], Pr=c["Pr"], U=c["U"],
                     precision=c["precision"], pattern=c["pattern"], seed=seed, noise_amp=0.0,
                     periodic_x=c["periodic_x"])


# ---- the model, as far as the initial fields and the 64-bit statement need it -----------------------
E2 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
E3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
      (1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1),
      (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)]


def _model(c):
    """Velocity sets, weights and relaxation rates (M1G scheme) of one lattice."""
    m = {"d3": c["dim"] == 3}
    L = float(c["ny"])
    m["L"], m["tau"] = L, 0.5 + c["U"] * math.sqrt(3.0) * L * math.sqrt(3.0 * c["Pr"] / c["Ra"])
    m["nu"] = (m["tau"] - 0.5) / 3.0
    m["kappa"] = m["nu"] / c["Pr"]
    m["gb"] = c["Ra"] * m["nu"] * m["kappa"] / L ** 3
    m["s_nu"] = 1.0 / m["tau"]
    m["s_q"] = 8.0 * (2.0 * m["tau"] - 1.0) / (8.0 * m["tau"] - 1.0)
    m["e"], m["eT"] = (E3, E3[:7]) if m["d3"] else (E2, E2[:5])
    by_speed = [1 / 3, 1 / 18, 1 / 36] if m["d3"] else [4 / 9, 1 / 9, 1 / 36]
    m["w"] = [by_speed[sum(abs(x) for x in v)] for v in m["e"]]
    m["wT"] = [0.25] + [0.125] * 6 if m["d3"] else [1 / 3] + [1 / 6] * 4
    m["qk"] = 1.0 / (0.5 + (4.0 * m["kappa"] if m["d3"] else 3.0 * m["kappa"]))
    m["geq"] = 4.0 if m["d3"] else 3.0
    return m


def _fields(c, seed):
    """A convecting state: populations in equilibrium with two rolls and a noisy temperature profile.
    Tensors on the GPU: f, g as (q, nz, ny, nx), scalars as (nz, ny, nx)."""
    m = _model(c)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
    rng = random.Random(seed)
    shape = (c["nz"], c["ny"], c["nx"])
    z, y, x = ((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n for n in shape)
    z, y, x = z[:, None, None], y[None, :, None], x[None, None, :]
    amp = rng.uniform(0.03, 0.05)
    sy, dsy = torch.sin(math.pi * y) ** 2, math.pi * torch.sin(2 * math.pi * y) / c["ny"]
    if c["periodic_x"]:
        ph = rng.uniform(0.0, 2 * math.pi)
        px, dpx = torch.sin(2 * math.pi * x + ph), 2 * math.pi * torch.cos(2 * math.pi * x + ph) / c["nx"]
    else:
        px, dpx = torch.sin(math.pi * x) ** 2, math.pi * torch.sin(2 * math.pi * x) / c["nx"]
    A = amp * c["ny"] / math.pi
    one = torch.ones(shape, device="cuda", dtype=torch.float64)
    if m["d3"]:
        wz, dz = torch.sin(math.pi * z) ** 2, math.pi * torch.sin(2 * math.pi * z) / c["nz"]
        wx = 1.0 if c["periodic_x"] else torch.sin(math.pi * x) ** 2
        u = one * (A * px * dsy * wz)
        v = one * (-A * dpx * sy * wz - 0.5 * A * dz * sy * wx)
        w = one * (0.5 * A * wz * dsy * wx)
    else:
        u, v, w = one * (A * px * dsy), one * (-A * dpx * sy), torch.zeros(shape, device="cuda", dtype=torch.float64)
    T = one * (0.5 - y + 0.2 * torch.sin(math.pi * y) * px)
    T += 1e-3 * (2.0 * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) - 1.0)
    u2 = u * u + v * v + w * w
    f = torch.empty((len(m["e"]),) + shape, device="cuda", dtype=torch.float64)
    g = torch.empty((len(m["eT"]),) + shape, device="cuda", dtype=torch.float64)
    for a, (ex, ey, ez) in enumerate(m["e"]):
        eu = ex * u + ey * v + ez * w
        f[a] = m["w"][a] * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * u2)
    for a, (ex, ey, ez) in enumerate(m["eT"]):
        g[a] = m["wT"][a] * T * (1.0 + m["geq"] * (ex * u + ey * v + ez * w))
    return {"f": f, "g": g, "rho": one, "u": u, "v": v, "w": w, "T": T, "Bx_prev": u * T, "By_prev": v * T,
            "Bz_prev": w * T, "Fy": m["gb"] * T}


def _host_state(c, seed):
    """The fields as a caller holds them: host arrays in Fortran layout (direction fastest)."""
    names = ["f", "g", "rho", "u", "v", "T", "Bx_prev", "By_prev"] + (["w", "Bz_prev"] if c["dim"] == 3 else ["Fy"])
    s = _fields(c, seed)
    out = {}
    for k in names:
        t = s.pop(k)
        t = t.permute(1, 2, 3, 0).contiguous() if t.dim() == 4 else t
        out[k] = (t if c["dim"] == 3 else t[0]).cpu().numpy()
    return out


def _lattice(c, seed):
    lat = lbmgpu.Lattice(_params(c, seed))
    lat.initial()
    return lat


def _load(lat, host):
    for k, a in host.items():
        lat.set_state(k, a)


def prepare(case, seed):
    if case["kind"] in ("batch", "streams"):
        group = lbmgpu.Ensemble() if case["kind"] == "batch" else StreamBatch()
        lats = []
        for n, c in enumerate(_member_cases(case)):
            lat = _lattice(c, seed + n)
            _load(lat, _host_state(c, seed * 1000 + n))
            lat.step(1)  # the step that reads loaded fields, which a member takes by itself
            group.add(lat)
            lats.append(lat)
        return {"case": case, "group": group, "lats": lats}
    lat = _lattice(case, seed)
    host = _host_state(case, seed)
    if case["kind"] == "job":
        return {"case": case, "lat": lat, "host": host}
    _load(lat, host)
    return {"case": case, "lat": lat}


def _read_back(case):
    """The fields of the solution that come back; the largest lattices are looked at through the
    temperature and the vertical velocity, a job through its temperature."""
    if case["kind"] == "job":
        return ("T",)
    if case["nx"] * case["ny"] * case["nz"] > 8e6:
        return ("T", "v")
    return ("T", "u", "v", "w") if case["dim"] == 3 else ("T", "u", "v")


def run(state):
    case = state["case"]
    dt = DTYPES[case["precision"]]
    if case["kind"] in ("batch", "streams"):
        group = state["group"]
        group.step(case["steps"])
        group.sync()
        return {"nu_re": np.array([lat.calNuRe() for lat in state["lats"]], dtype=dt),
                "T": [lat.get_state("T").astype(dt, copy=False) for lat in state["lats"]]}
    lat = state["lat"]
    if case["kind"] == "job":
        _load(lat, state["host"])
        lat.step(case["steps"])
        T = lat.get_state("T")
        return {"T": T.astype(dt, copy=False), "nu_re": np.array(lat.calNuRe(), dtype=dt)}
    if case["kind"] == "stages":
        for _ in range(case["steps"]):
            lat.stage_step()
    else:
        lat.step(case["steps"])
    out = {"nu_re": np.array(lat.calNuRe(), dtype=dt)}
    for k in _read_back(case):
        out[k] = lat.get_state(k).astype(dt, copy=False)
    return out


def work(case):
    """Populations read and written once per coupled cell update, and the fields that come back;
    615 (3D) or 250 (2D) floating-point operations per cell update."""
    total = {"bytes": 0.0, "flops": 0.0}
    for c in _member_cases(case) if case["kind"] in ("batch", "streams") else [case]:
        cells = c["nx"] * c["ny"] * c["nz"]
        pops = 26 if c["dim"] == 3 else 14
        total["bytes"] += 2.0 * pops * ESIZE[c["precision"]] * cells * c["steps"] + 8.0 * cells
        if case["kind"] == "job":
            total["bytes"] += 8.0 * (pops + 8) * cells
        total["flops"] += (615.0 if c["dim"] == 3 else 250.0) * cells * c["steps"]
    return total


# ---- the same steps in 64 bits, from the model's equations -------------------------------------------
def _rows(e, thermal, d3):
    """Rows of the moment matrix as polynomials of the velocities."""
    rows = []
    for x, y, z in e:
        s = x * x + y * y + z * z
        if thermal:
            rows.append([1, x, y, z, 7 * s - 6, 3 * x * x - s, y * y - z * z] if d3 else
                        [1, x, y, 5 * s - 4, x * x - y * y])
        elif d3:
            p, q = 3 * x * x - s, y * y - z * z
            rows.append([1, 19 * s - 30, (21 * s * s - 53 * s + 24) / 2, x, (5 * s - 9) * x, y, (5 * s - 9) * y, z,
                         (5 * s - 9) * z, p, (3 * s - 5) * p, q, (3 * s - 5) * q, x * y, y * z, x * z, q * x,
                         (z * z - x * x) * y, (x * x - y * y) * z])
        else:
            rows.append([1, 3 * s - 4, 4.5 * s * s - 10.5 * s + 4, x, (3 * s - 5) * x, y, (3 * s - 5) * y,
                         x * x - y * y, x * y])
    return torch.tensor(rows, dtype=torch.float64, device="cuda").T.contiguous()


def _stream(post, e, periodic_x, wall_sign, wall_term):
    """Streaming with the walls half way between cells: of the faces that a population's source lies
    beyond, the last of x, y, z decides.  wall_term: added at the two y walls (low, high)."""
    out = torch.empty_like(post)
    n = post.shape[1:]
    for a, v in enumerate(e):
        out[a] = torch.roll(post[a], shifts=(v[2], v[1], v[0]), dims=(0, 1, 2))
        opp = e.index((-v[0], -v[1], -v[2]))
        for axis, dim in ((0, 2), (1, 1), (2, 0)):
            if v[axis] == 0 or (axis == 2 and n[0] == 1):
                continue
            here = 0 if v[axis] > 0 else n[dim] - 1
            if axis == 0 and periodic_x:
                out[a].select(dim, here).copy_(post[a].select(dim, n[dim] - 1 - here))
            elif axis == 1:
                out[a].select(dim, here).copy_(wall_sign * post[opp].select(dim, here) + wall_term[0 if here == 0 else 1])
            else:
                out[a].select(dim, here).copy_(post[opp].select(dim, here))
    return out


def _exact_solve(c, seed, steps):
    m, s = _model(c), _fields(c, seed)
    d3, e, eT, gb, snu, sq = m["d3"], m["e"], m["eT"], m["gb"], m["s_nu"], m["s_q"]
    M, N = _rows(e, False, d3), _rows(eT, True, d3)
    Mi, Ni = torch.linalg.inv(M), torch.linalg.inv(N)
    f, g, rho, u, v, w, T = (s[k] for k in ("f", "g", "rho", "u", "v", "w", "T"))
    B = [s["Bx_prev"], s["By_prev"], s["Bz_prev"]]
    del s
    sg = 1.0 - 0.5 * m["qk"]
    shape = T.shape
    ex, ey, ez = (torch.tensor([x[i] for x in e], dtype=torch.float64, device="cuda") for i in range(3))
    for _ in range(steps):
        Fy = rho * gb * T  # the reference temperature is zero
        k = (M @ f.reshape(len(e), -1)).reshape(f.shape)
        uF = v * Fy

        def relax(i, eq, rate, source):
            k[i] += -rate * (k[i] - eq) + (1.0 - 0.5 * rate) * source

        if d3:
            u2 = u * u + v * v + w * w
            p, q = rho * (2 * u * u - v * v - w * w), rho * (v * v - w * w)
            relax(1, rho * (-11 + 19 * u2), snu, 38 * uF)
            relax(2, rho * (3 - 5.5 * u2), snu, -11 * uF)
            relax(4, -2 / 3 * rho * u, sq, 0.0)
            k[5] += Fy
            relax(6, -2 / 3 * rho * v, sq, -2 / 3 * Fy)
            relax(8, -2 / 3 * rho * w, sq, 0.0)
            relax(9, p, snu, -2 * uF)
            relax(10, -0.5 * p, snu, uF)
            relax(11, q, snu, 2 * uF)
            relax(12, -0.5 * q, snu, -uF)
            relax(13, rho * u * v, snu, u * Fy)
            relax(14, rho * v * w, snu, w * Fy)
            relax(15, rho * u * w, snu, 0.0)
            for i in (16, 17, 18):
                relax(i, 0.0, sq, 0.0)
        else:
            u2 = u * u + v * v
            relax(1, rho * (-2 + 3 * u2), snu, 6 * uF)
            relax(2, rho * (1 - 3 * u2), snu, -6 * uF)
            relax(4, -rho * u, sq, 0.0)
            k[5] += Fy
            relax(6, -rho * v, sq, -Fy)
            relax(7, rho * (u * u - v * v), snu, -2 * uF)
            relax(8, rho * u * v, snu, u * Fy)
        f = _stream((Mi @ k.reshape(len(e), -1)).reshape(f.shape), e, c["periodic_x"], 1.0, (0.0, 0.0))
        del k
        flat = f.reshape(len(e), -1)
        rho = flat.sum(0).reshape(shape)
        if d3:
            Fy = rho * gb * T
        u, v, w = ((d @ flat).reshape(shape) for d in (ex, ey, ez))
        u, v, w = u / rho, (v + 0.5 * Fy) / rho, w / rho
        n = (N @ g.reshape(len(eT), -1)).reshape(g.shape)
        for i, x in enumerate((u, v, w) if d3 else (u, v)):
            b = x * T
            n[1 + i] += -m["qk"] * (n[1 + i] - b) + sg * (b - B[i])
            B[i] = b
        if d3:
            n[4] = -0.75 * T
            n[5:] = 0.0
        else:
            n[3] = T * (-2.0 / 3.0)
            n[4] = 0.0
        wall = 2.0 * m["wT"][1] * 0.5
        g = _stream((Ni @ n.reshape(len(eT), -1)).reshape(g.shape), eT, c["periodic_x"], -1.0, (wall, -wall))
        T = g.sum(0)
    nu = float((v * T).mean()) * m["L"] / m["kappa"] + 1.0
    re = math.sqrt(float((u * u + v * v + w * w).mean())) * m["L"] / m["nu"]
    fields = {"T": T, "u": u, "v": v, "w": w}
    return {k: (t if d3 else t[0]).cpu().numpy() for k, t in fields.items()}, (nu, re)


def exact(case, seed):
    group = case["kind"] in ("batch", "streams")
    members = _member_cases(case) if group else [case]
    if sum(c["nx"] * c["ny"] * c["nz"] for c in members) * case["steps"] > EXACT_CELL_STEPS:
        return None
    if len(members) * case["steps"] > 4000:
        members = members[:max(1, 4000 // case["steps"])]  # many small lattices: the first of them
    if group:
        got = [_exact_solve(c, seed * 1000 + n, 1 + case["steps"]) for n, c in enumerate(members)]
        whole = len(got) == case["members"]
        return {"nu_re": np.array([x[1] for x in got]) if whole else None, "T": [x[0]["T"] for x in got]}
    fields, nu_re = _exact_solve(case, seed, case["steps"])
    return {"nu_re": np.array(nu_re), **{k: fields[k] for k in _read_back(case)}}
