"""Performance cases of the lattice Boltzmann engine: the work its users run.

A case is a dict of plain values; `prepare` builds on the GPU what a program
holds before the call (populations or initial fields, ping-pong buffers,
workspaces), `run` makes one pass through the public entry points of
lb-cube_b200/lbcube.py and returns its whole result. A pass of the stepping
cases is a chunk of time steps between two outputs, because that is how every
driver uses the step launchers: the buffers alternate and the initial state is
kept, so a pass can be repeated. `exact` repeats a pass in FP64 with plain torch.

Kinds of work:
  fluid     collide-stream steps (step_async)
  monitored equilibrium initialisation, steps, the step that also reduces the
            diagnostics, and the macroscopic output fields
  shifted   encode to 16-bit storage, steps on it, decode
  reactive  fluid + A + B -> C steps with the statistics appended to a device
            table every `every` steps (every = 0: no statistics)
  scalar    a fluid step and a passive scalar step, or the two-launch reaction
            (`species` 1 or 2), the sequence of the reference's drivers
  ke_grad   checkpointed gradient of the final kinetic energy
  re_grad   checkpointed gradient of the mean product
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

sys.path.insert(0, os.path.abspath("lb-cube_b200"))
import lbcube  # noqa: E402

Q_OF = {"D2Q9": 9, "D3Q19": 19, "D3Q27": 27}
SCALAR_Q = {"D2Q9": 5, "D3Q19": 7, "D3Q27": 7}
DTYPE = {"float": torch.float32, "double": torch.float64}


def listed():
    return [
        # A small 2-D study (a laptop-sized box, FP64 as the drivers default to): launches count.
        {"name": "d2q9_f64_bgk_128", "kind": "fluid", "lattice": "D2Q9", "real": "double", "op": "BGK",
         "nx": 128, "ny": 128, "nz": 1, "tau": 0.6, "steps": 50},
        # The Taylor-Green validation box of lbm_sim (64^3 FP64 BGK), which fits in L2.
        {"name": "d3q19_f64_bgk_64", "kind": "fluid", "lattice": "D3Q19", "real": "double", "op": "BGK",
         "nx": 64, "ny": 64, "nz": 64, "tau": 0.6, "steps": 20},
        # The headline turbulence box.
        {"name": "d3q19_f32_trt_256", "kind": "fluid", "lattice": "D3Q19", "real": "float", "op": "TRT",
         "nx": 256, "ny": 256, "nz": 256, "tau": 0.55, "steps": 10},
        # A channel-like box with odd extents, as a user's geometry gives them.
        {"name": "d3q19_f32_mrt_odd", "kind": "fluid", "lattice": "D3Q19", "real": "float", "op": "MRT",
         "nx": 201, "ny": 130, "nz": 75, "tau": 0.55, "steps": 10},
        # The 27-velocity lattice with its own MRT operator, at the size of a resolved TGV study.
        {"name": "d3q27_f32_mrt_128", "kind": "fluid", "lattice": "D3Q27", "real": "float", "op": "MRT",
         "nx": 128, "ny": 128, "nz": 128, "tau": 0.55, "steps": 10},
        # A run watched from the host: initial state, steps, blow-up guard and output fields.
        {"name": "monitored_f32_trt_160", "kind": "monitored", "lattice": "D3Q19", "real": "float", "op": "TRT",
         "nx": 160, "ny": 160, "nz": 160, "tau": 0.55, "steps": 10},
        # 16-bit storage at the headline size, from FP32 populations and back.
        {"name": "shifted_f16_trt_256", "kind": "shifted", "lattice": "D3Q19", "fmt": "f16s", "op": "TRT",
         "nx": 256, "ny": 256, "nz": 256, "tau": 0.55, "steps": 20},
        # 16-bit storage on a box whose rows are no multiple of 8 cells.
        {"name": "shifted_q15_mrt_100", "kind": "shifted", "lattice": "D3Q19", "fmt": "q15s", "op": "MRT",
         "nx": 100, "ny": 90, "nz": 111, "tau": 0.55, "steps": 20},
        # The 2-D reactive-mixing configuration, statistics every 10 steps.
        {"name": "reactive_d2q9_mrt_1024", "kind": "reactive", "lattice": "D2Q9", "real": "float", "op": "MRT",
         "nx": 1024, "ny": 1024, "nz": 1, "tau": 0.6, "tau_c": 0.62, "k": 4e-5, "steps": 30, "every": 10},
        # A passive tracer in a 3-D flow, fluid and scalar launched in turn (odd rows).
        {"name": "scalar_f32_trt_135", "kind": "scalar", "lattice": "D3Q19", "real": "float", "op": "TRT",
         "nx": 135, "ny": 128, "nz": 90, "tau": 0.55, "tau_c": 0.8, "species": 1, "steps": 10},
        # The kinetic-energy gradient at its configured 128^3, over two checkpoint segments.
        {"name": "ke_grad_f32_bgk_128", "kind": "ke_grad", "lattice": "D3Q19", "real": "float", "op": "BGK",
         "nx": 128, "ny": 128, "nz": 128, "tau": 0.56, "steps": 20, "interval": 10},
        # The reactive gradient at its configured 192^3 with FP16 stored states.
        {"name": "re_grad_f16_trt_192", "kind": "re_grad", "lattice": "D3Q19", "real": "float", "op": "TRT",
         "storage": "f16s", "nx": 192, "ny": 192, "nz": 192, "tau": 0.55, "tau_c": 0.8, "k": 0.02,
         "steps": 12, "interval": 6},
    ]


# ---- draws -----------------------------------------------------------------------
DRAW_BYTES = 12e9  # at most this much work per drawn pass (the largest listed case has 4 times as much)


def _box(rng, dims, lo, hi, multiple=1):
    """Extents of a box of lo .. hi cells (log-uniform), any aspect up to about 1 : 5."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = cells ** (1.0 / dims)
    e = [max(4, int(round(side * math.exp(rng.uniform(-0.8, 0.8) / (dims - 1))))) for _ in range(dims - 1)]
    last = max(3, int(round(cells / math.prod(e))))
    e.append(last)
    e[0] = max(multiple, e[0] // multiple * multiple)
    if multiple == 1 and rng.random() < 0.4:  # the round sizes people pick
        e[0] = max(8, (e[0] + 8) // 16 * 16)
    return e + [1] if dims == 2 else e


def draw(rng):
    kind = rng.choices(["fluid", "monitored", "shifted", "reactive", "scalar", "ke_grad", "re_grad"],
                       [5, 1, 3, 2, 1, 1, 1])[0]
    lat = rng.choices(["D2Q9", "D3Q19", "D3Q27"], [2, 5, 2])[0]
    dims = 2 if lat == "D2Q9" else 3
    real = rng.choice(["float", "float", "double"])
    op = rng.choice(["BGK", "TRT", "MRT", "RLBM"])
    c = {"kind": kind, "lattice": lat, "real": real, "op": op, "tau": round(rng.uniform(0.53, 0.9), 3)}
    hi, multiple = 1.6e7, 1
    if kind == "shifted":
        c["fmt"] = rng.choice(["f16s", "f16s", "bf16s", "e3m12s", "q15s"])
        del c["real"]
        multiple = 4
    if kind in ("reactive", "scalar", "re_grad"):
        c["tau_c"] = round(rng.uniform(0.55, 1.0), 3)
        c["k"] = round(math.exp(rng.uniform(math.log(1e-4), math.log(5e-2))), 6)
        hi = 6e6
    if kind == "scalar":
        c["species"] = rng.choice([1, 2])
    elif kind != "fluid" and kind != "monitored" and kind != "shifted" and op == "RLBM":
        c["op"] = "TRT"
    if kind in ("ke_grad", "re_grad"):
        if lat == "D3Q27":
            c["lattice"] = "D3Q19"
        hi = 1.5e6
        c["steps"] = rng.randint(6, 14)
        c["interval"] = rng.randint(3, 8)
        if kind == "re_grad":
            c["storage"] = rng.choice(["native", "native", "f16s", "bf16s"])
            if c["storage"] != "native":
                c["real"] = "float"
    else:
        c["steps"] = rng.randint(8, 40)
    c["nx"], c["ny"], c["nz"] = _box(rng, dims, 4e3, hi, multiple)
    if kind == "reactive":
        c["every"] = rng.choice([0, 4, 10])
    while work(c)["bytes"] > DRAW_BYTES and c["steps"] > 4:
        c["steps"] -= 1
    while work(c)["bytes"] > DRAW_BYTES:
        axis = "ny" if dims == 2 else "nz"
        c[axis] = max(3, c[axis] // 2)
    return c


# ---- inputs ----------------------------------------------------------------------
def _lattice(name):
    """Velocities and weights in the [Q, Z, Y, X] population order of the interface."""
    axes3 = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
    edges = [(1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1),
             (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)]
    corners = [(x, y, z) for z in (1, -1) for y in (1, -1) for x in (1, -1)]
    axes2 = [(1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0)]
    rest = [(0, 0, 0)]
    if name == "D2Q9":
        return rest + axes2 + [(1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)], [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
    if name == "D3Q19":
        return rest + axes3 + edges, [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
    if name == "D3Q27":
        return rest + axes3 + edges + corners, [8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8
    if name == "D2Q5":
        return rest + axes2, [1 / 3] + [1 / 6] * 4
    return rest + axes3, [1 / 4] + [1 / 8] * 6  # D3Q7


def _fields(case, seed):
    """rho, u (Taylor-Green plus seeded noise) and the species' concentrations
    (interleaved blocks of 0 and 1 in 3-D, two halves in 2-D, a little noise)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dims = 2 if case["lattice"] == "D2Q9" else 3
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = DTYPE[case.get("real", "float")]
    x, y, z = (torch.arange(n, device="cuda", dtype=torch.float32) * (2 * math.pi / n) for n in (nx, ny, nz))
    sx, cx, sy, cy = x.sin()[None, None, :], x.cos()[None, None, :], y.sin()[None, :, None], y.cos()[None, :, None]
    cz = z.cos()[:, None, None] if dims == 3 else torch.ones(1, 1, 1, device="cuda")
    u = torch.zeros(dims, nz, ny, nx, device="cuda")
    u[0] = 0.05 * sx * cy * cz
    u[1] = -0.05 * cx * sy * cz
    u += 1e-3 * torch.randn(u.shape, generator=gen, device="cuda")
    rho = 1.0 + 1e-3 * torch.randn((nz, ny, nx), generator=gen, device="cuda")
    out = {"rho": rho.to(dt).contiguous(), "u": u.to(dt).contiguous()}
    if case["kind"] in ("reactive", "scalar", "re_grad"):
        if dims == 2:
            a = (torch.arange(ny, device="cuda") * 2 >= ny).float()[None, :, None].expand(nz, ny, nx)
        else:
            bx, by, bz = (torch.arange(n, device="cuda") // 16 for n in (nx, ny, nz))
            a = ((bx[None, None, :] + by[None, :, None] + bz[:, None, None]) % 2).float()
        noise = 0.01 * torch.rand((nz, ny, nx), generator=gen, device="cuda")
        out["a"] = (a + noise).to(dt).contiguous()
        out["b"] = (1.0 - a + noise).to(dt).contiguous()
    return out


def _equilibrium(lattice, rho, u):
    c, w = _lattice(lattice)
    dims = u.shape[0]
    usq = (u * u).sum(0)
    out = torch.empty((len(c),) + rho.shape, dtype=rho.dtype, device=rho.device)
    for i, (ci, wi) in enumerate(zip(c, w)):
        cu = sum(ci[d] * u[d] for d in range(dims) if ci[d]) if any(ci) else torch.zeros_like(rho)
        if lattice in ("D2Q5", "D3Q7"):
            out[i] = wi * rho * (1 + cu * (3.0 if lattice == "D2Q5" else 4.0))
        else:
            out[i] = wi * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq)
    return out


def _scalar_name(case):
    return "D2Q5" if case["lattice"] == "D2Q9" else "D3Q7"


def prepare(case, seed):
    s = {"case": case, "n": (case["nx"], case["ny"], case["nz"])}
    f = _fields(case, seed)
    kind, lat = case["kind"], case["lattice"]
    dev = "cuda"
    if kind in ("ke_grad", "re_grad"):
        s.update(f)
        grad = (case["lattice"], case["real"], *s["n"], case["steps"], case["interval"])
        if kind == "ke_grad":
            size = lbcube.ke_gradient_workspace_bytes(*grad)
        else:
            size = lbcube.reactive_gradient_workspace_bytes(*grad, storage=case["storage"])
            s["grad_a"], s["grad_b"] = torch.empty_like(f["a"]), torch.empty_like(f["b"])
        s["size"] = size
        s["work"] = torch.empty(size, dtype=torch.uint8, device=dev)
        s["out"] = torch.empty(4 if kind == "re_grad" else 2, dtype=torch.float64, device=dev)
        s["grad_u"] = torch.empty_like(f["u"])
        return s
    if kind == "monitored":
        s.update(f)
        s["size"] = lbcube.diagnostics_partials_bytes(lat, *s["n"])
        s["partials"] = torch.empty(s["size"] // 8, dtype=torch.float64, device=dev)
        s["diag"] = torch.empty(5, dtype=torch.float64, device=dev)
        s["density"], s["speed"], s["velocity"] = (torch.empty_like(f[k]) for k in ("rho", "rho", "u"))
        s["f"] = [torch.empty((Q_OF[lat],) + f["rho"].shape, dtype=f["rho"].dtype, device=dev) for _ in range(2)]
        return s
    f0 = _equilibrium(lat, f["rho"], f["u"])
    if kind == "shifted":
        s["f0"], s["back"] = f0, torch.empty_like(f0)
        s["h"] = [torch.empty(f0.shape, dtype=torch.int16, device=dev) for _ in range(2)]
        return s
    s["f0"] = f0
    s["f"] = [torch.empty_like(f0) for _ in range(2)]
    if kind in ("reactive", "scalar"):
        still = torch.zeros_like(f["u"])
        for name in ("a", "b"):
            s[name + "0"] = _equilibrium(_scalar_name(case), f[name], still)
            s[name] = [torch.empty_like(s[name + "0"]) for _ in range(2)]
    if kind == "reactive" and case["every"]:
        s["rows"] = case["steps"] // case["every"]
        s["size"] = lbcube.stats_partials_bytes(lat, *s["n"])
        s["partials"] = torch.empty(s["size"] // 8, dtype=torch.float64, device=dev)
        s["table"] = torch.zeros(max(1, s["rows"]), 8, dtype=torch.float64, device=dev)
        s["row"] = torch.zeros(1, dtype=torch.int64, device=dev)
    return s


# ---- one pass --------------------------------------------------------------------
def _run_fluid(s, c, n):
    omega, cur = 1.0 / c["tau"], s["f0"]
    for i in range(c["steps"]):
        nxt = s["f"][i % 2]
        lbcube.check(lbcube.step_async(c["lattice"], c["real"], c["op"], cur, nxt, *n, omega))
        cur = nxt
    return cur


def _run_monitored(s, c, n):
    omega, (cur, nxt) = 1.0 / c["tau"], s["f"]
    lbcube.check(lbcube.init_equilibrium_async(c["lattice"], c["real"], s["rho"], s["u"], cur, *n))
    for _ in range(c["steps"] - 1):
        lbcube.check(lbcube.step_async(c["lattice"], c["real"], c["op"], cur, nxt, *n, omega))
        cur, nxt = nxt, cur
    lbcube.check(lbcube.step_diagnostics_async(c["lattice"], c["real"], c["op"], cur, nxt, *n, omega, s["partials"],
                                               s["size"], s["diag"], 0.4))
    lbcube.check(lbcube.macro_fields_async(c["lattice"], c["real"], nxt, *n, s["density"], s["velocity"], s["speed"]))
    return [nxt, s["diag"], s["density"], s["velocity"], s["speed"]]


def _run_shifted(s, c, n):
    omega, (cur, nxt) = 1.0 / c["tau"], s["h"]
    lbcube.check(lbcube.encode_shifted_async(c["lattice"], c["fmt"], "float", s["f0"], cur, *n))
    for _ in range(c["steps"]):
        lbcube.check(lbcube.step_shifted_async(c["lattice"], c["fmt"], c["op"], cur, nxt, *n, omega))
        cur, nxt = nxt, cur
    lbcube.check(lbcube.decode_shifted_async(c["lattice"], c["fmt"], "float", cur, s["back"], *n))
    return s["back"]


def _run_reactive(s, c, n):
    lat, real, omega, omega_c = c["lattice"], c["real"], 1.0 / c["tau"], 1.0 / c["tau_c"]
    f, a, b = s["f0"], s["a0"], s["b0"]
    every = c["every"]
    if every:
        s["row"].zero_()
    for i in range(c["steps"]):
        nf, na, nb = s["f"][i % 2], s["a"][i % 2], s["b"][i % 2]
        if every and (i + 1) % every == 0:
            lbcube.check(lbcube.fluid_reaction_ab_async(lat, real, c["op"], f, nf, a, na, b, nb, *n, omega, omega_c,
                                                        c["k"], s["partials"], s["size"]))
            lbcube.check(lbcube.reactive_stats_append_async(lat, real, *n, c["k"], s["partials"], s["size"], s["table"],
                                                            s["table"].shape[0], s["row"]))
        else:
            lbcube.check(lbcube.fluid_reaction_ab_async(lat, real, c["op"], f, nf, a, na, b, nb, *n, omega, omega_c,
                                                        c["k"]))
        f, a, b = nf, na, nb
    return [f, a, b] + ([s["table"]] if every else [])


def _run_scalar(s, c, n):
    lat, real, omega, omega_c = c["lattice"], c["real"], 1.0 / c["tau"], 1.0 / c["tau_c"]
    f, a, b = s["f0"], s["a0"], s["b0"]
    for i in range(c["steps"]):
        nf, na, nb = s["f"][i % 2], s["a"][i % 2], s["b"][i % 2]
        lbcube.check(lbcube.step_async(lat, real, c["op"], f, nf, *n, omega))
        if c["species"] == 1:
            lbcube.check(lbcube.scalar_step_async(lat, real, a, na, nf, *n, omega_c))
        else:
            lbcube.check(lbcube.reaction_ab_async(lat, real, a, na, b, nb, nf, *n, omega_c, c["k"]))
        f, a, b = nf, na, nb
    return [f, a] if c["species"] == 1 else [f, a, b]


def _run_ke_grad(s, c, n):
    lbcube.check(lbcube.ke_gradient_async(c["lattice"], c["real"], c["op"], s["rho"], s["u"], *n, c["tau"], c["steps"],
                                          c["interval"], s["work"], s["size"], s["out"], s["grad_u"]))
    return [s["out"], s["grad_u"]]


def _run_re_grad(s, c, n):
    lbcube.check(lbcube.reactive_gradient_async(
        c["lattice"], c["real"], c["op"], "mean_product", s["rho"], s["u"], s["a"], s["b"], *n, c["tau"], c["tau_c"],
        c["k"], c["steps"], c["interval"], s["work"], s["size"], s["out"], s["grad_a"], s["grad_b"], s["grad_u"],
        storage=c["storage"]))
    return [s["out"], s["grad_a"], s["grad_b"], s["grad_u"]]


_RUN = {"fluid": _run_fluid, "monitored": _run_monitored, "shifted": _run_shifted, "reactive": _run_reactive,
        "scalar": _run_scalar, "ke_grad": _run_ke_grad, "re_grad": _run_re_grad}


def run(state):
    return _RUN[state["case"]["kind"]](state, state["case"], state["n"])


# ---- what a pass cannot do without --------------------------------------------------
def work(case):
    """Every step reads and writes each population once; a gradient also
    recomputes all but its last checkpoint segment and takes each step back
    (state read, adjoint state read and written)."""
    cells = case["nx"] * case["ny"] * case["nz"]
    q, sq, dims = Q_OF[case["lattice"]], SCALAR_Q[case["lattice"]], 2 if case["lattice"] == "D2Q9" else 3
    e = 8 if case.get("real") == "double" else 4
    n, kind = case["steps"], case["kind"]
    flops = (2 * q * q if case["op"] == "MRT" else 14 * q) * n
    if kind == "fluid":
        per = 2 * q * e * n
    elif kind == "monitored":
        per = 2 * q * e * n + (1 + dims + q) * e + (q + 2 + dims) * e
    elif kind == "shifted":
        per = 4 * q * n + 2 * (4 + 2) * q
    elif kind == "reactive":
        per, flops = 2 * (q + 2 * sq) * e * n, flops + 24 * sq * n
    elif kind == "scalar":
        per = (2 * q + q + 2 * sq * case["species"]) * e * n
        flops += 12 * sq * case["species"] * n
    else:
        pops = q + (2 * sq if kind == "re_grad" else 0)
        stored = 2 if case.get("storage", "native") != "native" else e
        again = (n - 1) // case["interval"] * (case["interval"] - 1)
        per = (n + again) * 2 * pops * stored + n * pops * (stored + 2 * e) + (1 + 2 * dims) * e
        flops *= 3
    return {"bytes": float(cells * per), "flops": float(cells * flops)}


# ---- the same pass in 64 bits -------------------------------------------------------
def _pull(f, lattice):
    """Every population streamed one link along its velocity (periodic)."""
    c, _ = _lattice(lattice)
    return torch.stack([torch.roll(f[i], shifts=(ci[2], ci[1], ci[0]), dims=(0, 1, 2)) for i, ci in enumerate(c)])


def _macro(f, lattice):
    c, _ = _lattice(lattice)
    dims = 2 if lattice == "D2Q9" else 3
    rho = f.sum(0)
    return rho, torch.stack([sum(ci[d] * f[i] for i, ci in enumerate(c) if ci[d]) for d in range(dims)]) / rho


def _orthogonal(lattice):
    """The moment polynomials of the D2Q9 and D3Q19 MRT operators on their velocity sets."""
    c = np.array(_lattice(lattice)[0], float)
    x, y, z = c.T
    s = (c * c).sum(1)
    if lattice == "D2Q9":
        rows = [1 + 0 * s, 3 * s - 4, 4 - 10.5 * s + 4.5 * s * s, x, (3 * s - 5) * x, y, (3 * s - 5) * y, x * x - y * y, x * y]
    else:
        xx, ww = 3 * x * x - s, y * y - z * z
        rows = [1 + 0 * s, 19 * s - 30, (21 * s * s - 53 * s + 24) / 2, x, (5 * s - 9) * x, y, (5 * s - 9) * y,
                z, (5 * s - 9) * z, xx, ww, x * y, y * z, x * z, (3 * s - 5) * xx, (3 * s - 5) * ww, ww * x,
                (z * z - x * x) * y, (x * x - y * y) * z]
    return np.array(rows)


def _mrt(f, lattice, omega):
    rho, u = _macro(f, lattice)
    if lattice == "D3Q27":  # moments of the product basis 1, c, 3 c^2 - 2, relaxed towards those of the equilibrium
        c = np.array(_lattice(lattice)[0])
        basis = lambda k, v: np.ones_like(v) if k == 0 else (v if k == 1 else 3 * v * v - 2)  # noqa: E731
        orders = [(a, b, d) for a in range(3) for b in range(3) for d in range(3)]
        m = np.array([basis(a, c[:, 0]) * basis(b, c[:, 1]) * basis(d, c[:, 2]) for a, b, d in orders], float)
        rate = np.zeros((27, 27))
        for i, o in enumerate(orders):
            if sum(o) < 2:
                continue
            if o in ((1, 1, 0), (1, 0, 1), (0, 1, 1)):
                rate[i, i] = -1.0  # the shear rate
            elif o in ((2, 0, 0), (0, 2, 0), (0, 0, 2)):
                for p in ((2, 0, 0), (0, 2, 0), (0, 0, 2)):  # trace with 1.19, the rest with the shear rate
                    rate[i, orders.index(p)] += 1.19 / 3
            else:
                rate[i, i] = 1.1 if sum(o) == 3 and max(o) == 2 else 1.2
        inverse = m.T / (m * m).sum(1)
        shear = np.diag((rate == -1.0).diagonal().astype(float))
        diag = [orders.index(p) for p in ((2, 0, 0), (0, 2, 0), (0, 0, 2))]
        for i in diag:
            for j in diag:
                shear[i, j] += (1.0 if i == j else 0.0) - 1 / 3
        fixed = np.where(rate == -1.0, 0.0, rate)
        to = lambda k: torch.tensor(k, dtype=f.dtype, device=f.device)  # noqa: E731
        op = to(inverse @ fixed @ m) + omega * to(inverse @ shear @ m)
        neq = (f - _equilibrium(lattice, rho, u)).reshape(27, -1)
        return f - (op @ neq).reshape(f.shape)
    mat = _orthogonal(lattice)
    m = (torch.tensor(mat, dtype=f.dtype, device=f.device) @ f.reshape(f.shape[0], -1)).reshape(f.shape)
    usq = (u * u).sum(0)
    if lattice == "D2Q9":
        j = rho * u
        eq = {1: -2 * rho + 3 * rho * usq, 2: rho - 3 * rho * usq, 4: -j[0], 6: -j[1],
              7: rho * (u[0] ** 2 - u[1] ** 2), 8: rho * u[0] * u[1]}
        rate = {1: 1.63, 2: 1.14, 4: 1.92, 6: 1.92, 7: omega, 8: omega}
    else:
        x2, y2, z2 = u[0] ** 2, u[1] ** 2, u[2] ** 2
        zero = torch.zeros_like(rho)
        eq = {1: -11 * rho + 19 * rho * usq, 2: 3 * rho - 5.5 * rho * usq, 4: -2 / 3 * rho * u[0], 6: -2 / 3 * rho * u[1],
              8: -2 / 3 * rho * u[2], 9: 3 * rho * (2 * x2 - y2 - z2), 10: rho * (y2 - z2), 11: rho * u[0] * u[1],
              12: rho * u[1] * u[2], 13: rho * u[0] * u[2], **{k: zero for k in range(14, 19)}}
        rate = {k: omega if 9 <= k <= 13 else 1.0 for k in eq}
    m = torch.stack([m[k] - rate[k] * (m[k] - eq[k]) if k in eq else m[k] for k in range(m.shape[0])])
    inverse = torch.tensor(mat.T / (mat * mat).sum(1), dtype=f.dtype, device=f.device)
    return (inverse @ m.reshape(m.shape[0], -1)).reshape(f.shape)


def _rlbm(f, lattice, omega):
    """Recursive regularised collision: second- and third-order Hermite terms of the non-equilibrium stress."""
    c, w = _lattice(lattice)
    dims = 2 if lattice == "D2Q9" else 3
    rho, u = _macro(f, lattice)
    fe = _equilibrium(lattice, rho, u)
    neq = f - fe
    pi = {(a, b): sum(ci[a] * ci[b] * neq[i] for i, ci in enumerate(c) if ci[a] * ci[b]) for a in range(dims)
          for b in range(a, dims)}
    p = lambda a, b: pi[(min(a, b), max(a, b))]  # noqa: E731
    third = lambda a, b, d: u[a] * p(b, d) + u[b] * p(a, d) + u[d] * p(a, b)  # noqa: E731
    del neq, f
    out = torch.empty_like(fe)
    for i, (ci, wi) in enumerate(zip(c, w)):
        delta = lambda a, b: 1 / 3 if a == b else 0.0  # noqa: E731
        acc = sum((ci[a] * ci[b] - delta(a, b)) * p(a, b) for a in range(dims) for b in range(dims))
        h = lambda a, b: ci[a] * ci[a] * ci[b] - ci[b] / 3  # noqa: E731  (a a b)
        if lattice == "D3Q19":
            for (e, g), (k, l) in (((0, 1), (2, 1)), ((2, 0), (1, 0)), ((1, 2), (0, 2))):
                hp, hm = h(e, g) + h(k, l), h(e, g) - h(k, l)
                if hp:
                    acc = acc + 3 * hp * (third(e, e, g) + third(k, k, l))
                if hm:
                    acc = acc + hm * (third(e, e, g) - third(k, k, l))
        else:
            for a in range(dims):
                for b in range(dims):
                    hab = h(a, b) if a != b else ci[a] ** 3 - ci[a]
                    if hab:
                        acc = acc + (1 if a == b else 3) * hab * third(a, a, b)
            if dims == 3 and ci[0] * ci[1] * ci[2]:
                acc = acc + 6 * ci[0] * ci[1] * ci[2] * third(0, 1, 2)
        out[i] = fe[i] + (1 - omega) * wi * 4.5 * acc
    return out


def _collide(f, lattice, op, tau):
    omega = 1 / tau
    if op == "MRT":
        return _mrt(f, lattice, omega)
    if op == "RLBM":
        return _rlbm(f, lattice, omega)
    rho, u = _macro(f, lattice)
    neq = f - _equilibrium_grad(lattice, rho, u)
    if op == "BGK":
        return f - omega * neq
    c, _ = _lattice(lattice)
    opposite = [c.index(tuple(-k for k in ci)) for ci in c]
    omega_minus = 1 / (0.25 / (tau - 0.5) + 0.5)
    back = neq[opposite]
    return f - 0.5 * omega * (neq + back) - 0.5 * omega_minus * (neq - back)


def _equilibrium_grad(lattice, rho, u):
    """_equilibrium without writes in place, for autograd."""
    c, w = _lattice(lattice)
    usq = (u * u).sum(0)
    out = []
    for ci, wi in zip(c, w):
        cu = sum(ci[d] * u[d] for d in range(u.shape[0]) if ci[d]) if any(ci) else 0.0 * rho
        if lattice in ("D2Q5", "D3Q7"):
            out.append(wi * rho * (1 + cu * (3.0 if lattice == "D2Q5" else 4.0)))
        else:
            out.append(wi * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq))
    return torch.stack(out)


def _scalar(g, lattice, u, tau_c, source):
    sl = "D2Q5" if lattice == "D2Q9" else "D3Q7"
    _, w = _lattice(sl)
    eq = _equilibrium_grad(sl, g.sum(0), u)
    wt = torch.tensor(w, dtype=g.dtype, device=g.device).reshape(-1, 1, 1, 1)
    return g + (eq - g) / tau_c + wt * source


def _source(ca, cb, k):
    """Exact A + B -> C batch step; -expm1 keeps the difference of close concentrations."""
    diff = cb - ca
    same = diff.abs() < 1e-9
    d = torch.where(same, torch.ones_like(diff), diff)
    # a' = a d e / (b - a e) with e = exp(-k d), b - a e = d - a (e - 1)
    em1 = torch.expm1(-k * d)
    return torch.where(same, ca / (1 + k * ca), ca * d * (em1 + 1) / (d - ca * em1)) - ca


def _coupled(f, a, b, case, tau, tau_c, k):
    lat = case["lattice"]
    sl = _scalar_name(case)
    f = _collide(_pull(f, lat), lat, case["op"], tau)
    _, u = _macro(f, lat)
    a, b = _pull(a, sl), _pull(b, sl)
    src = _source(a.sum(0), b.sum(0), k)
    return f, _scalar(a, lat, u, tau_c, src), _scalar(b, lat, u, tau_c, src)


def _seconds(case):
    """A generous estimate of exact()'s time: FP64 passes over the populations."""
    cells, q = case["nx"] * case["ny"] * case["nz"], Q_OF[case["lattice"]]
    heavy = 5 if case["op"] == "RLBM" else 1
    grad = 4 if case["kind"] in ("ke_grad", "re_grad") else 1
    return cells * q * case["steps"] * 8.0 * 40 * heavy * grad / 2.5e12


def exact(case, seed):
    if _seconds(case) > 15:
        return None
    fields = _fields(case, seed)
    x = {k: v.double() for k, v in fields.items()}
    kind, lat, op, tau = case["kind"], case["lattice"], case["op"], case["tau"]
    if kind in ("ke_grad", "re_grad"):
        return _exact_gradient(case, x)
    if kind == "monitored":
        f = _equilibrium(lat, x["rho"], x["u"])
    else:
        f = _equilibrium(lat, fields["rho"], fields["u"]).double()
    del fields
    with torch.no_grad():
        if kind in ("fluid", "monitored", "shifted"):
            del x
            for _ in range(case["steps"]):
                f = _collide(_pull(f, lat), lat, op, tau)
            if kind != "monitored":
                return f
            rho, u = _macro(f, lat)
            s2 = (u * u).sum(0)
            diag = torch.stack([rho.sum(), (0.5 * rho * s2).sum(), s2.max().sqrt(), 0 * rho.sum(), 0 * rho.sum()])
            return [f, diag, rho, u, s2.sqrt()]
        sl = _scalar_name(case)
        real = DTYPE[case["real"]]
        a, b = (_equilibrium(sl, x[n].to(real), torch.zeros_like(x["u"], dtype=real)).double() for n in ("a", "b"))
        rows = []
        for i in range(case["steps"]):
            if kind == "reactive":
                f, a, b = _coupled(f, a, b, case, tau, case["tau_c"], case["k"])
                if case["every"] and (i + 1) % case["every"] == 0:
                    ca, cb = a.sum(0), b.sum(0)
                    ma, mb, mab = ca.mean(), cb.mean(), (ca * cb).mean()
                    cov = mab - ma * mb
                    rows.append(torch.stack([ma, mb, (ca * ca).mean() - ma * ma, (cb * cb).mean() - mb * mb, cov,
                                             cov / (ma * mb), case["k"] * mab, case["k"] * ma * mb]))
            else:
                f = _collide(_pull(f, lat), lat, op, tau)
                _, u = _macro(f, lat)
                a, b = _pull(a, sl), _pull(b, sl)
                src = _source(a.sum(0), b.sum(0), case["k"]) if case["species"] == 2 else 0.0
                a = _scalar(a, lat, u, case["tau_c"], src)
                if case["species"] == 2:
                    b = _scalar(b, lat, u, case["tau_c"], src)
        if kind == "scalar":
            return [f, a] if case["species"] == 1 else [f, a, b]
        table = torch.stack(rows) if rows else torch.zeros(1, 8, dtype=torch.float64, device="cuda")
        return [f, a, b] + ([table] if case["every"] else [])


def _exact_gradient(case, x):
    lat, op = case["lattice"], case["op"]
    leaf = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True)  # noqa: E731
    u0, tau = x["u"].requires_grad_(True), leaf(case["tau"])
    f = _equilibrium_grad(lat, x["rho"], u0)
    if case["kind"] == "ke_grad":
        for _ in range(case["steps"]):
            f = checkpoint(lambda g: _collide(_pull(g, lat), lat, op, tau), f, use_reentrant=False)
        rho, u = _macro(f, lat)
        obj = (0.5 * rho * (u * u).sum(0)).sum()
        obj.backward()
        return [torch.stack([obj.detach(), tau.grad]), u0.grad]
    sl = _scalar_name(case)
    a0, b0, tau_c, k = x["a"].requires_grad_(True), x["b"].requires_grad_(True), leaf(case["tau_c"]), leaf(case["k"])
    a, b = _equilibrium_grad(sl, a0, u0), _equilibrium_grad(sl, b0, u0)
    for _ in range(case["steps"]):
        f, a, b = checkpoint(lambda g, p, q: _coupled(g, p, q, case, tau, tau_c, k), f, a, b, use_reentrant=False)
    obj = a0.mean() - a.sum(0).mean()
    obj.backward()
    return [torch.stack([obj.detach(), k.grad, tau.grad, tau_c.grad]), a0.grad, b0.grad, u0.grad]
