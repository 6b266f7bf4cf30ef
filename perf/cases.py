"""The workloads whose speed this framework is judged by, through its public entry points.

listed() names them, draw() gives more of the same ranges, prepare() makes what a program holds before the
call, run() is one call of it, exact() restates the result in 64-bit torch.  Every case is a stretch of a
machining simulation as its callers drive it: the engine steps the workpiece in sub-cycles, reads the metrics and
takes the particle records (kind "frame"), couples them to other solvers (kind "coupling"), runs many workpieces
at once (kinds "sweep" and "served") or moves a whole state through host memory (kind "exchange").

Inputs: a box workpiece whose particles are jittered inside their octant of the cell, a seeded velocity and
temperature field around the cutting zone, and for "developed" states a shear zone at the edge of yield with
plastic strain, damage and heat, as a cut leaves it; in a sweep the seed varies the cutting speed and material.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "edegpredict-engine-rotary_b200"))
from mpm_b200 import Batch, Server, Solver, capi as A, workpiece as W  # noqa: E402

MATERIALS = {"4340": W.AISI_4340, "ti64": W.TI_6AL_4V}
SHEAR_DEFAULTS = dict(asb_enabled=1, asb_critical_rate=1e4, asb_taylor_quinney=0.9, asb_max_temp_ratio=0.9,
                      asb_touch_rise=0.5)
RECORD = 504                                   # bytes of a particle record (63 doubles)
PX, PV, PEXT, PT, PF, PFP, PC, PS, PEPS = 0, 3, 9, 16, 17, 26, 35, 44, 56


def _box(kind, wx, wy, wz, steps, material="4340", ppc=8, precision="f32", boundary="sticky", developed=False,
         options=""):
    return dict(kind=kind, wx=wx, wy=wy, wz=wz, steps=steps, material=material, ppc=ppc, precision=precision,
                boundary=boundary, developed=developed, options=options)


def listed():
    return [
        # one sub-step of a small workpiece and the metrics after it: the engine's finest interleaving
        dict(_box("frame", 12, 10, 8, 1), name="tiny_step"),
        # the small plain workpiece (64x32x32 cells, AISI 4340, cylinder), one frame of 8 sub-steps
        dict(_box("frame", 64, 32, 32, 8), name="small_frame"),
        # the precision study's workpiece (128x64x64 cells, Ti-6Al-4V, wedge)
        dict(_box("frame", 128, 64, 64, 8, material="ti64"), name="medium_frame"),
        # the plain large workpiece (256x128x128 cells, 33.5 M particles)
        dict(_box("frame", 256, 128, 128, 8, material="ti64"), name="large_frame"),
        # the drop-in solver's tool boundary: tool samples set each frame and rasterised each step; an odd box,
        # 5 particles per cell, a developed cut
        dict(_box("frame", 53, 37, 29, 5, ppc=5, boundary="raster", developed=True), name="ragged_raster"),
        # 64-bit state: the precision study's reference runs
        dict(_box("frame", 64, 32, 32, 4, precision="f64", developed=True), name="double_frame"),
        # adiabatic shear heating and grid heat conduction in every step, node sums with atomics (the launch
        # configuration's faster, not bit-reproducible mode)
        dict(_box("frame", 64, 32, 32, 8, developed=True, options="heat"), name="heat_frame"),
        # particle-side tool contact with friction in every step, slip boundary
        dict(_box("frame", 64, 32, 32, 8, boundary="slip", developed=True, options="contact"), name="contact_frame"),
        # another solver writes the particle records between single steps (drag and cooling of chips)
        dict(_box("coupling", 48, 40, 30, 1), name="coupled_step"),
        # a parameter sweep of uneven workpieces in one batch, 10 steps a call from a captured graph
        dict(kind="sweep", count=48, lo=12, hi=40, shapes=7, steps=10, name="sweep"),
        # solve requests served to completion: admission, ticks, results
        dict(kind="served", count=10, lo=10, hi=24, shapes=5, steps=40, name="served"),
        # a whole state in from host arrays and out again around a few steps (the callers without device records)
        dict(_box("exchange", 32, 24, 20, 4, developed=True), name="host_exchange"),
    ]


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "raster", "f64", "heat", "contact", "coupling", "sweep", "served",
                       "exchange"])
    if kind == "sweep":
        return dict(kind="sweep", count=rng.randint(8, 64), lo=rng.randint(8, 14), hi=rng.randint(18, 40),
                    shapes=rng.randint(0, 10 ** 6), steps=rng.randint(2, 20))
    if kind == "served":
        return dict(kind="served", count=rng.randint(2, 16), lo=rng.randint(6, 10), hi=rng.randint(12, 28),
                    shapes=rng.randint(0, 10 ** 6), steps=rng.randint(10, 60))
    most = {"frame": 4.0e6, "raster": 4e5, "f64": 3e5, "heat": 6e5, "contact": 6e5, "coupling": 3e5,
            "exchange": 4e4}[kind]
    cells = math.exp(rng.uniform(math.log(600.0), math.log(most)))
    ax, ay = rng.uniform(1.0, 3.0), rng.uniform(0.8, 2.0)
    wz = max(6, round((cells / (ax * ay)) ** (1 / 3)))
    wx, wy = max(6, round(ax * wz)), max(6, round(ay * wz))
    c = _box("frame", wx, wy, wz, rng.randint(1, 12), material=rng.choice(["4340", "ti64"]), ppc=rng.randint(4, 8))
    if kind == "frame":
        c["boundary"] = rng.choice(["sticky", "sticky", "slip"])
        c["developed"] = wx * wy * wz < 3e5 and rng.random() < 0.5
    elif kind == "raster":
        c.update(boundary="raster", developed=True)
    elif kind == "f64":
        c.update(precision="f64", developed=True, steps=rng.randint(1, 6))
    elif kind == "heat":
        c.update(options="heat", developed=True)
    elif kind == "contact":
        c.update(options="contact", boundary="slip", developed=True)
    elif kind == "coupling":
        c.update(kind="coupling", steps=1)
    else:
        c.update(kind="exchange", developed=True, steps=rng.randint(1, 8))
    return c


# ------------------------------------------------------------------ inputs

def _workpiece(c):
    """The workpiece of a box case: parameters, tool and box as the package's configurations lay them out."""
    ti = c["material"] == "ti64"
    mode = {"sticky": A.TOOL_SDF_STICKY, "slip": A.TOOL_SDF_SLIP, "raster": A.TOOL_RASTER}[c["boundary"]]
    w = W.make_case((c["wx"], c["wy"], c["wz"]), 2e-5 if ti else 5e-5, c["ppc"], MATERIALS[c["material"]],
                    "wedge" if ti else "cylinder", doc=5e-5 if ti else 1e-4, speed=2.5 if ti else 1.67,
                    radius=3e-4 if ti else 5e-4, steps=c["steps"], tool_mode=mode,
                    tool_x_cells=min(16.0, c["wx"] / 3.0),
                    precision=A.PREC_F64 if c["precision"] == "f64" else A.PREC_F32)
    if c["boundary"] == "raster":
        w["tool"]["samples"] = W.tool_samples(w)
    p = w["params"]
    if c["options"] == "heat":
        p.update(SHEAR_DEFAULTS, heat_conduction=1, thermal_conductivity=42.6)
    if c["options"] == "contact":
        p.update(contact_every=1, contact_radius=0.5 * p["dx"], contact_friction=0.3, contact_heat_partition=0.5)
    return w


def _field(w, pos, seed):
    """Velocity and temperature around the cutting zone at positions pos [n, 3], and the zone's weight."""
    p, t = w["params"], w["tool"]
    dx = p["dx"]
    g = torch.Generator(device=pos.device).manual_seed(seed % (1 << 31) + 1)
    rnd = torch.randn(pos.shape[0], 4, generator=g, device=pos.device, dtype=torch.float64)
    ahead = (pos[:, 0] - t["position"][0] - t["radius"]) / dx
    below = (pos[:, 2] - (t["position"][2] - t["radius"])) / dx
    zone = torch.exp(-((0.7 * ahead - 0.7 * below) / 4.0) ** 2 - ((ahead + below) / 24.0) ** 2)
    speed = t["velocity"][0]
    v = 0.01 * speed * rnd[:, :3]
    v[:, 0] += 0.5 * speed * zone
    v[:, 2] += 0.3 * speed * zone
    T = p["Tamb"] + 2.0 * rnd[:, 3].abs() + 400.0 * zone
    return v, T, zone


def _developed(w, seed, device):
    """A full particle state as a cut leaves it, every field in 64 bits."""
    p = w["params"]
    pos, status = _points(w, device)
    v, T, zone = _field(w, pos, seed)
    n = pos.shape[0]
    g = torch.Generator(device=device).manual_seed(seed % (1 << 31) + 2)
    u = torch.rand(n, 2, generator=g, device=device, dtype=torch.float64)
    mu = p["E"] / (2.0 * (1.0 + p["nu"]))
    elastic = 0.7 * p["jc_A"] / (math.sqrt(3.0) * mu) * zone * (0.9 + 0.2 * u[:, 0])
    plastic = 0.15 * zone
    F = torch.eye(3, dtype=torch.float64, device=device).repeat(n, 1, 1)
    Fp = F.clone()
    F[:, 0, 2] = elastic + plastic
    Fp[:, 0, 2] = plastic
    eps = plastic / math.sqrt(3.0)
    v[status == A.FIXED] = 0.0
    t = w["tool"]
    above = pos[:, 2] > t["position"][2] + t["tip_dz"]         # damage below the tool tip is a chip's
    return dict(x=pos, v=v, T=T, F=F, Fp=Fp, C=torch.zeros_like(F), eps=eps, edot=1e4 * zone,
                D=0.1 * zone * above * u[:, 1] * p["D_th"], status=status)


def _points(w, device):
    """The particles of the box generator: Philox4x32-10 points, each in its own octant of the cell, those inside
    the tool left out."""
    p, b = w["params"], w["box"]
    c0, c1, ppc = b["c0"], b["c1"], b["ppc"]
    wx, wy, wz = (c1[a] - c0[a] for a in range(3))
    cand = torch.arange(wx * wy * wz * ppc, device=device, dtype=torch.int64)
    cell, k = cand // ppc, cand % ppc
    m = 0xFFFFFFFF
    k0, k1 = b["seed"] & m, (b["seed"] >> 32) & m
    r = [cell & m, k & m, torch.full_like(cell, b["instance"]), torch.zeros_like(cell)]
    for _ in range(10):
        a, d = r[0] * 0xD2511F53, r[2] * 0xCD9E8D57
        r = [((d >> 32) & m) ^ r[1] ^ k0, d & m, ((a >> 32) & m) ^ r[3] ^ k1, a & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    octant = torch.tensor([0, 7, 3, 4, 5, 2, 6, 1], device=device)[k]
    at = [cell % wx, (cell // wx) % wy, cell // (wx * wy)]
    pos = torch.empty(cand.numel(), 3, device=device, dtype=torch.float64)
    for a in range(3):
        off = 0.5 * ((octant >> a) & 1).double() + 0.5 * ((r[a] >> 8).double() / 16777216.0)
        pos[:, a] = p["origin"][a] + ((c0[a] + at[a]).double() + off) * p["dx"]
    status = torch.where(at[2] < b["fixed_layers"], A.FIXED, A.ACTIVE)
    keep = _tool_distance(w["tool"], pos[:, 0], pos[:, 2], w["tool"]["position"][0], w["tool"]["position"][2])[0] > 0
    return pos[keep], status[keep]


def _on_host(st):
    h = {k: t.cpu().numpy() for k, t in st.items()}
    n = len(h["status"])
    out = {a: np.ascontiguousarray(h["x"][:, i]) for i, a in enumerate("xyz")}
    out.update({"v" + a: np.ascontiguousarray(h["v"][:, i]) for i, a in enumerate("xyz")})
    out.update(F=h["F"].reshape(n, 9), Fp=h["Fp"].reshape(n, 9), C=h["C"].reshape(n, 9), plastic_strain=h["eps"],
               strain_rate=h["edot"], temperature=h["T"], damage=h["D"], status=h["status"].astype(np.int32),
               id=np.arange(n, dtype=np.int32))
    return out


def _sweep(c, seed):
    """Workpieces of uneven size and material; the seed varies the cutting speed and the flow stress."""
    rng, vary = np.random.default_rng(c["shapes"]), np.random.default_rng(seed % (1 << 31))
    ws = [W.config3_case(rng, i, cells_lo=c["lo"], cells_hi=c["hi"], steps=c["steps"],
                         ppc=8 if c["kind"] == "served" else None) for i in range(c["count"])]
    for w in ws:
        f = vary.uniform(0.8, 1.25, 2)
        w["tool"]["velocity"] = (w["tool"]["velocity"][0] * f[0], 0.0, 0.0)
        w["params"]["jc_A"] *= f[1]
    return ws


def _capacity(w):
    b = w["box"]
    return int(np.prod([b["c1"][a] - b["c0"][a] for a in range(3)])) * b["ppc"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        ws = _sweep(case, seed)
        s = Batch([W.to_mpm_params(w) for w in ws], [_capacity(w) for w in ws])
        s.set_launch_config(use_graph=True)
        n = []
        for i, w in enumerate(ws):
            b = w["box"]
            n.append(s.init_box_i(i, b["c0"], b["c1"], b["ppc"], b["seed"], b["instance"], b["fixed_layers"], b["T0"],
                                  tool=w["tool"]))
        return dict(kind=kind, s=s, n=n, dt=[w["dt"] for w in ws], steps=case["steps"],
                    buf=torch.empty(sum(n), RECORD // 8, dtype=torch.float64, device="cuda"))
    if kind == "served":
        s = Server(hbm_budget_bytes=6 << 30, max_chunk=20)
        return dict(kind=kind, s=s, ws=_sweep(case, seed), steps=case["steps"])
    w = _workpiece(case)
    stream = torch.cuda.Stream()
    s = Solver(W.to_mpm_params(w), _capacity(w), stream=stream.cuda_stream)
    if case["options"] == "heat":
        s.set_launch_config(deterministic=False)
    b = w["box"]
    state = dict(kind=kind, s=s, w=w, dt=w["dt"], steps=case["steps"], stream=stream, frame=0,
                 raster=case["boundary"] == "raster")
    if kind == "exchange":
        s.set_tool(w["tool"])
        state["host"] = _on_host(_developed(w, seed, "cuda"))
        return state
    if case["developed"]:
        st = _developed(w, seed, "cuda")
        n = st["status"].numel()
        s.set_tool(w["tool"])
        s.upload(_on_host(st))
        state["buf"] = torch.empty(n, RECORD // 8, dtype=torch.float64, device="cuda")
    else:
        n = s.init_box(b["c0"], b["c1"], b["ppc"], b["seed"], b["instance"], b["fixed_layers"], b["T0"],
                       tool=w["tool"])
        buf = state["buf"] = torch.empty(n, RECORD // 8, dtype=torch.float64, device="cuda")
        s.export_aos_device(buf.data_ptr(), n * RECORD)
        with torch.cuda.stream(stream):
            v, T, _ = _field(w, buf[:, PX:PX + 3], seed)
            buf[:, PV:PV + 3], buf[:, PT] = v, T
        s.import_aos(buf.data_ptr(), A.AOS_VELOCITY | A.AOS_TEMPERATURE, nbytes=n * RECORD)
    if kind == "coupling":
        s.export_aos_device(state["buf"].data_ptr(), n * RECORD)
    torch.cuda.synchronize()
    return state


# ------------------------------------------------------------------ the calls

METRICS = ("mass", "kinetic", "internal_elastic", "thermal", "max_temperature", "max_von_mises", "mean_plastic_strain")
COUNTS = ("n_active", "n_chip", "n_fixed", "n_inactive")


def _metrics(m):
    out = {k: float(m[k]) for k in METRICS}
    out["momentum"] = np.array(m["momentum"])
    out["counts"] = np.array([m[k] for k in COUNTS])
    return out


def _records(buf):
    """The fields of exported particle records."""
    ints = buf.view(torch.int32)
    return dict(position=buf[:, PX:PX + 3], velocity=buf[:, PV:PV + 3], temperature=buf[:, PT],
                F=buf[:, PF:PF + 9], Fp=buf[:, PFP:PFP + 9], C=buf[:, PC:PC + 9], stress=buf[:, PS:PS + 6],
                plastic_strain=buf[:, PEPS], strain_rate=buf[:, PEPS + 1], damage=buf[:, PEPS + 2],
                residual=buf[:, PEPS + 3], status=ints[:, 121])


def run(state):
    kind, s = state["kind"], state["s"]
    if kind == "sweep":
        s.step_all(state["dt"], state["steps"])
        m = [s.metrics_i(0), s.metrics_i(len(state["n"]) - 1)]
        buf, at = state["buf"], 0
        for i, n in enumerate(state["n"]):
            A.check(A.lib().mpm_batch_export_aos(s.h, i, buf.data_ptr() + at * RECORD, n * RECORD), s.h)
            at += n
        return [_records(buf), [_metrics(x) for x in m]]
    if kind == "served":
        ids = [s.submit(w, state["steps"] + 7 * (i % 4)) for i, w in enumerate(state["ws"])]
        while s.tick() or s.stats()["queued"]:
            pass
        got = [s.poll(i) for i in ids]
        return {k: np.array([x["metrics"][k] for x in got]) for k in METRICS + COUNTS + ("momentum",)}
    if kind == "exchange":
        s.upload(state["host"])
        s.step(state["dt"], state["steps"])
        m = s.metrics()
        out = s.download(fields=("x", "y", "z", "vx", "vy", "vz", "F", "Fp", "C", "stress", "plastic_strain",
                                 "strain_rate", "temperature", "damage", "residual_stress", "status", "id"))
        s.reset_clock()
        s.set_tool(state["w"]["tool"])
        return [_host_fields(out), _metrics(m)]
    buf = state["buf"]
    if kind == "coupling":
        with torch.cuda.stream(state["stream"]):
            chips = 2e-3 * state["w"]["params"]["particle_mass"] / state["dt"]
            torch.mul(buf[:, PV:PV + 3], -chips, out=buf[:, PEXT:PEXT + 3])
            buf[:, PT].mul_(0.999).add_(1e-3 * state["w"]["params"]["Tamb"])
        s.import_aos(buf.data_ptr(), A.AOS_WRITABLE, nbytes=buf.numel() * 8)
    if state["raster"]:
        t = dict(state["w"]["tool"])
        at = state["frame"] * state["steps"] * state["dt"]
        t["position"] = tuple(t["position"][a] + t["velocity"][a] * at for a in range(3))
        s.set_tool(t)
    s.step(state["dt"], state["steps"])
    state["frame"] += 1
    m = s.metrics()
    s.export_aos_device(buf.data_ptr(), buf.numel() * 8)
    return [_records(buf), _metrics(m)]


def _host_fields(o):
    return dict(position=np.stack([o["x"], o["y"], o["z"]], 1), velocity=np.stack([o["vx"], o["vy"], o["vz"]], 1),
                F=o["F"], Fp=o["Fp"], C=o["C"], stress=o["stress"], plastic_strain=o["plastic_strain"],
                strain_rate=o["strain_rate"], temperature=o["temperature"], damage=o["damage"],
                residual=o["residual_stress"], status=o["status"])


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """A step reads and writes each particle's moving state once and each grid node twice; a call also reads and
    writes velocity, C and stress once, and its records, host arrays or results are written (and read) once.  About
    1400 floating operations a particle and step."""
    if case["kind"] in ("sweep", "served"):
        ws = _sweep(case, 1)
        steps = [case["steps"] + (7 * (i % 4) if case["kind"] == "served" else 0) for i in range(len(ws))]
        e = 4
    else:
        ws, steps, e = [_workpiece(dict(case, boundary="sticky"))], [case["steps"]], 4
        e = 8 if case["precision"] == "f64" else 4
    b = f = 0.0
    for w, k in zip(ws, steps):
        p, n = w["params"], _capacity(w)
        read, wrote = 7 * 4 * e + 1, 5 * 4 * e
        b += n * k * (read + wrote) + k * 2 * 4 * e * p["nx"] * p["ny"] * p["nz"] + n * (8 + 6) * 4 * e
        f += 1400.0 * n * k
        if case["kind"] == "exchange":
            b += n * (32 + 43) * 8
        elif case["kind"] == "coupling":
            b += n * 2 * RECORD
        elif case["kind"] != "served":
            b += n * RECORD
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times what the fields differ by when the node sums take another order (the launch configuration's
    pass size and atomics: up to 6e-6, in C and the plastic strain; 64-bit state 5e-14).  A particle that crosses a
    threshold of the model one step apart may differ by more than the rest."""
    if case.get("precision") == "f64":
        return {"rel": 1e-11, "max": 1e-6, "differ": 1e-4}
    return {"rel": 3e-5, "max": 0.02, "differ": 1e-4}


# ------------------------------------------------------------------ the step in 64 bits

def _tool_distance(t, x, z, px, pz):
    """Signed distance to the tool (a cylinder along y or a rounded wedge) and its outward normal (x, z)."""
    qx, qz = x - px, z - pz
    if t["shape"] == A.SHAPE_CYLINDER_Y:
        r = torch.sqrt(qx * qx + qz * qz)
        return r - t["radius"], qx / r.clamp_min(1e-300), qz / r.clamp_min(1e-300)
    sg, cg, sa, ca = math.sin(t["rake"]), math.cos(t["rake"]), math.sin(t["clearance"]), math.cos(t["clearance"])
    d1, d2 = cg * qx + sg * qz, -sa * qx - ca * qz
    s1, s2 = (cg * qz - sg * qx).clamp_min(0.0), (sa * qz - ca * qx).clamp_min(0.0)
    e1x, e1z, e2x, e2z = qx + s1 * sg, qz - s1 * cg, qx + s2 * ca, qz - s2 * sa
    l1, l2 = torch.sqrt(e1x * e1x + e1z * e1z), torch.sqrt(e2x * e2x + e2z * e2z)
    inside = (d1 <= 0) & (d2 <= 0)
    one = torch.ones_like(qx)
    first = l1 <= l2
    nx = torch.where(inside, torch.where(d1 >= d2, cg * one, -sa * one),
                     torch.where(first, e1x / l1.clamp_min(1e-300), e2x / l2.clamp_min(1e-300)))
    nz = torch.where(inside, torch.where(d1 >= d2, sg * one, -ca * one),
                     torch.where(first, e1z / l1.clamp_min(1e-300), e2z / l2.clamp_min(1e-300)))
    return torch.where(inside, torch.maximum(d1, d2), torch.minimum(l1, l2)) - t["radius"], nx, nz


class _Exact:
    """The material point step on torch tensors in 64 bits: quadratic B-spline APIC transfers, the grid update with
    the fixture and the tool, the Johnson-Cook return, and the options the cases use."""

    def __init__(self, w, st):
        self.w, self.p, self.st, self.step, self.time = w, w["params"], st, 0, 0.0
        n, dev = st["status"].numel(), st["x"].device
        zero = torch.zeros(n, dtype=torch.float64, device=dev)
        st.setdefault("F", torch.eye(3, dtype=torch.float64, device=dev).repeat(n, 1, 1))
        st.setdefault("Fp", st["F"].clone())
        st.setdefault("C", torch.zeros_like(st["F"]))
        for k in ("eps", "edot", "D"):
            st.setdefault(k, zero.clone())
        st["sig"], st["sres"] = torch.zeros_like(st["F"]), zero.clone()
        st["asb"] = torch.zeros(n, dtype=torch.int64, device=dev)
        p = self.p
        self.org = torch.tensor(p["origin"], dtype=torch.float64, device=dev)
        self.mu = p["E"] / (2 * (1 + p["nu"]))
        self.lam = p["E"] * p["nu"] / ((1 + p["nu"]) * (1 - 2 * p["nu"]))
        self.chunk = 2_000_000

    def _stencil(self, x):
        xi = (x - self.org) / self.p["dx"]
        base = torch.floor(xi - 0.5)
        d = xi - base
        wt = torch.stack([0.5 * (1.5 - d) ** 2, 0.75 - (d - 1) ** 2, 0.5 * (d - 0.5) ** 2], 2)
        dw = torch.stack([d - 1.5, -2 * (d - 1), d - 0.5], 2) / self.p["dx"]
        return base.long(), wt, dw

    def _offsets(self, x):
        base, wt, dw = self._stencil(x)
        nx, ny = self.p["nx"], self.p["ny"]
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    o = torch.tensor([i, j, k], device=x.device)
                    g = base + o
                    ww = wt[:, 0, i] * wt[:, 1, j] * wt[:, 2, k]
                    gw = torch.stack([dw[:, 0, i] * wt[:, 1, j] * wt[:, 2, k], wt[:, 0, i] * dw[:, 1, j] * wt[:, 2, k],
                                      wt[:, 0, i] * wt[:, 1, j] * dw[:, 2, k]], 1)
                    yield g[:, 0] + nx * (g[:, 1] + ny * g[:, 2]), ww, gw, self.org + g.double() * self.p["dx"] - x

    def _constitutive(self, s, dt):
        """Stress of the ACTIVE particles (with the reference's trial lower triangle for the force) and their
        plastic state, heat and damage."""
        p, st = self.p, s
        act = st["status"] == A.ACTIVE
        Fe = st["F"] @ torch.linalg.inv(st["Fp"])
        J = torch.linalg.det(Fe).clamp(0.9, 1.1)
        eye = torch.eye(3, dtype=torch.float64, device=J.device)
        sig = (self.mu / J)[:, None, None] * (Fe @ Fe.mT - eye) + (self.lam * (J - 1))[:, None, None] * eye
        p3 = sig.diagonal(dim1=1, dim2=2).sum(1) / 3
        dev = sig - p3[:, None, None] * eye
        q = torch.sqrt(1.5 * (dev * dev).sum((1, 2)))
        T = st["T"]
        Ts = ((T - p["Tamb"]) / max(p["Tm"] - p["Tamb"], 1.0)).clamp(0, 1)
        es = (st["edot"] / max(p["edot0"], 1e-12)).clamp_min(1e-5)
        Y = (p["jc_A"] + p["jc_B"] * st["eps"] ** p["jc_n"]) * (1 + p["jc_C"] * torch.log(es)) * (1 - Ts ** p["jc_m"])
        flow = act & (q > Y) & (q > 1e-12)
        dE = torch.where(flow, ((q - Y) / (3 * self.mu)).clamp_max(p["deps_cap"]), 0.0)
        sc = torch.where(flow, Y / q.clamp_min(1e-300), 1.0)
        upper = torch.triu(torch.ones_like(eye))
        sd = dev * (upper * sc[:, None, None] + (1 - upper))         # lower triangle keeps its trial value
        sym = torch.triu(sd) + torch.triu(sd, 1).mT
        full = sd + p3[:, None, None] * eye
        stored = sym + p3[:, None, None] * eye
        plastic = flow & (dE > 0)
        sn = torch.sqrt((sym * sym).sum((1, 2)))
        al = torch.where(plastic & (sn > 1e-12), 1.5 * dE / sn.clamp_min(1e-300), 0.0)
        Fp = (eye + al[:, None, None] * sd) @ st["Fp"]
        Fp = Fp / torch.linalg.det(Fp).clamp_min(1e-12).pow(1 / 3)[:, None, None]
        st["Fp"] = torch.where(plastic[:, None, None], Fp, st["Fp"])
        st["eps"] = st["eps"] + torch.where(plastic, dE, 0.0)
        heat = p["beta"] / max(p["rho_phys"] * p["cp"], 1e-12)
        st["T"] = torch.where(plastic, (T + (heat * Y * dE).clamp_max(p["dT_cap"])).clamp_max(p["Tm"]), T)
        ef = (p["D1"] + p["D2"] * torch.exp(p["D3"] * p3 / q.clamp_min(1e-12))) * \
            (1 + p["D4"] * torch.log(es.clamp_min(1.0))) * (1 + p["D5"] * Ts)
        hurt = plastic & (ef > 1e-12)
        st["D"] = st["D"] + torch.where(hurt, dE / ef.clamp_min(1e-300), 0.0)
        worn = hurt & (st["D"] > 0.7 * p["D_th"])
        f = torch.where(worn, ((p["D_th"] - st["D"]) / (0.3 * p["D_th"])).clamp(0, 1), 1.0)[:, None, None]
        st["sres"] = torch.where(worn, torch.maximum(st["sres"], torch.sqrt(1.5 * (sym * sym).sum((1, 2)))), st["sres"])
        st["sig"] = torch.where(act[:, None, None], f * stored, st["sig"])
        st["status"] = torch.where(hurt & (st["D"] >= p["D_th"]), A.CHIP, st["status"])
        pushes = act & (st["status"] == A.ACTIVE)
        V = p["particle_volume"]
        return torch.where(pushes[:, None, None], -dt * V * J[:, None, None] * f * full, 0.0)

    def _node_positions(self):
        p, dev = self.p, self.org.device
        i = torch.arange(p["nx"] * p["ny"] * p["nz"], device=dev)
        return (i % p["nx"]).double(), ((i // p["nx"]) % p["ny"]).double(), (i // (p["nx"] * p["ny"])).double()

    def _grid(self, g, dt, pose):
        p, t = self.p, self.w["tool"]
        m = g[:, 0]
        on = m > p["mass_threshold"]
        v = g[:, 1:4].clone()
        v[:, 2] += m * p["gravity_z"] * dt
        v = torch.where(on[:, None], v / m.clamp_min(1e-300)[:, None], 0.0)
        ix, iy, iz = self._node_positions()
        zr = iz * p["dx"] / p["fixture_thickness"]
        f = 1 / (1 + p["fixture_damping"] * (1 - zr) ** 2 * dt)
        f = torch.where(iz == 0, 0.0, torch.where(zr <= 1, f, torch.ones_like(zr)))
        v = v * f[:, None]
        tv = torch.tensor(t["velocity"], dtype=torch.float64, device=v.device)
        if t["mode"] == A.TOOL_RASTER:
            s = torch.tensor(np.asarray(t["samples"]), device=v.device)
            c = (s + torch.tensor(pose, dtype=torch.float64, device=v.device) - self.org) / p["dx"]
            c = (torch.sign(c) * torch.floor(c.abs() + 0.5)).long()
            mark = torch.zeros(v.shape[0], dtype=torch.bool, device=v.device)
            for a in range(8):
                q = c + torch.tensor([a & 1, (a >> 1) & 1, a >> 2], device=v.device)
                ok = ((q >= 0) & (q < torch.tensor([p["nx"], p["ny"], p["nz"]], device=v.device))).all(1)
                q = q[ok]
                mark[q[:, 0] + p["nx"] * (q[:, 1] + p["ny"] * q[:, 2])] = True
            return torch.where((on & mark)[:, None], tv, v)
        phi, nx, nz = _tool_distance(t, ix * p["dx"] + p["origin"][0], iz * p["dx"] + p["origin"][2], pose[0], pose[2])
        hit = on & (phi <= 0)
        if t["mode"] == A.TOOL_SDF_STICKY:
            return torch.where(hit[:, None], tv, v)
        nrm = torch.stack([nx, torch.zeros_like(nx), nz], 1)
        vn = ((v - tv) * nrm).sum(1).clamp_max(0.0)
        return v - torch.where(hit, vn, 0.0)[:, None] * nrm

    def _diffuse(self, g, dt):
        p = self.p
        shape = (p["nz"], p["ny"], p["nx"])
        m, tm = g[:, 0].view(shape), g[:, 4].view(shape)
        T = tm / m.clamp_min(1e-30)
        lap = torch.zeros_like(T)
        for a in range(3):
            d = T.diff(dim=a)
            n = T.shape[a]
            lap.narrow(a, 0, n - 1).add_(d)
            lap.narrow(a, 1, n - 1).sub_(d)
        c = p["thermal_conductivity"] / (p["rho_phys"] * p["cp"]) * dt / p["dx"] ** 2
        out = torch.where(m >= 1e-15, (T + c * lap).clamp_min(0.0), torch.where(m > 0, tm / m.clamp_min(1e-300), 0.0))
        return out.view(-1)

    def advance(self, steps, dt, force=None):
        p, t, st = self.p, self.w["tool"], self.st
        heat = bool(p.get("heat_conduction"))
        n = st["status"].numel()
        mass = p["particle_mass"]
        for k in range(steps):
            pose = [t["position"][a] + t["velocity"][a] * self.time for a in range(3)]
            g = torch.zeros(p["nx"] * p["ny"] * p["nz"], 5 if heat else 4, dtype=torch.float64, device=self.org.device)
            for lo in range(0, n, self.chunk):
                s = {q: a[lo:lo + self.chunk] for q, a in st.items()}
                cell = torch.floor((s["x"] - self.org) / p["dx"])
                far = torch.tensor([p["nx"] - 2, p["ny"] - 2, p["nz"] - 2], device=cell.device)
                s["status"] = torch.where(((cell < 1) | (cell >= far)).any(1), A.INACTIVE, s["status"])
                S = self._constitutive(s, dt)
                live, moves = s["status"] != A.INACTIVE, (s["status"] != A.INACTIVE) & (s["status"] != A.FIXED)
                ext = force[lo:lo + self.chunk] * dt if force is not None and k == 0 else None
                for idx, ww, gw, dp in self._offsets(s["x"]):
                    mom = ww[:, None] * mass * (s["v"] + (s["C"] @ dp[:, :, None])[:, :, 0]) + \
                        (S @ gw[:, :, None])[:, :, 0]
                    mom = torch.where(moves[:, None], mom, 0.0)
                    if ext is not None:
                        mom = mom + torch.where(live[:, None], ww[:, None] * ext, 0.0)
                    val = [torch.where(live, ww * mass, 0.0)[:, None], mom]
                    if heat:
                        val.append((val[0][:, 0] * s["T"])[:, None])
                    g.index_add_(0, torch.where(live, idx, 0), torch.cat(val, 1))
                for q in st:
                    st[q][lo:lo + self.chunk] = s[q]
            tn = self._diffuse(g, dt) if heat else None
            vel = self._grid(g, dt, pose)
            for lo in range(0, n, self.chunk):
                s = {q: a[lo:lo + self.chunk] for q, a in st.items()}
                moves = (s["status"] != A.INACTIVE) & (s["status"] != A.FIXED)
                v, B, L = torch.zeros_like(s["v"]), torch.zeros_like(s["C"]), torch.zeros_like(s["C"])
                ts, ws = torch.zeros_like(s["T"]), torch.zeros_like(s["T"])
                for idx, ww, gw, dp in self._offsets(s["x"]):
                    idx = torch.where(moves, idx, 0)
                    nv = vel[idx]
                    v += ww[:, None] * nv
                    B += (ww[:, None] * nv)[:, :, None] * dp[:, None, :]
                    L += nv[:, :, None] * gw[:, None, :]
                    if heat:
                        use = g[idx, 0] > 1e-18
                        ts += torch.where(use, ww * tn[idx], 0.0)
                        ws += torch.where(use, ww, 0.0)
                if heat:
                    s["T"] = torch.where(moves & (ws > 1e-8), (ts / ws.clamp_min(1e-300)).clamp(p["Tamb"], p["Tm"]),
                                         s["T"])
                chip = s["status"] == A.CHIP
                s["v"] = torch.where(moves[:, None], v, torch.where((s["status"] == A.FIXED)[:, None], 0.0, s["v"]))
                s["x"] = s["x"] + torch.where(moves[:, None], v * dt, 0.0)
                solid = moves & ~chip
                C = p["apic_dinv_factor"] / p["dx"] ** 2 * p["apic_decay"] * B
                s["C"] = torch.where(solid[:, None, None], C, s["C"])
                s["F"] = torch.where(solid[:, None, None], s["F"] + dt * (L @ s["F"]), s["F"])
                D = 0.5 * (L + L.mT)
                rate = torch.sqrt(2.0 / 3.0 * (D * D).sum((1, 2)))
                s["edot"] = torch.where(solid, rate, torch.where(chip, 0.0, s["edot"]))
                self._after_move(s, lo, dt, pose)
                for q in st:
                    st[q][lo:lo + self.chunk] = s[q]
            self.step += 1
            self.time += dt

    def _after_move(self, s, lo, dt, pose):
        p, t = self.p, self.w["tool"]
        if p.get("asb_enabled"):
            chip = s["status"] == A.CHIP
            warm = (s["status"] == A.ACTIVE) & (s["T"] > p["Tamb"] + p["asb_touch_rise"])
            fast = warm & (s["edot"] >= max(p["asb_critical_rate"] * 0.5, 5000.0))
            sg = s["sig"]
            dev = sg - sg.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] * torch.eye(3, device=sg.device)
            seq = torch.sqrt(1.5 * (dev * dev).sum((1, 2)))
            base = p["asb_taylor_quinney"] * seq * s["edot"] * dt / max(p["rho_phys"] * p["cp"], 1e-12)
            c = torch.where(fast, (s["asb"] + 1).clamp_max(10),
                            torch.where(warm, (s["asb"] - 1).clamp_min(0), torch.where(chip, 0, s["asb"])))
            ratio = (1 + 1.5 * (s["edot"] / max(p["asb_critical_rate"], 1.0) - 1)).clamp_max(2.5)
            inc = torch.where((s["edot"] > p["asb_critical_rate"]) & (c >= 3), base * ratio, base)
            cap = base.clamp_max(100.0)
            inc = torch.where((cap > 0) & (inc > cap), cap, inc)
            s["T"] = torch.where(fast, (s["T"] + inc).clamp_max(p["asb_max_temp_ratio"] * p["Tm"]), s["T"])
            s["asb"] = c
        if p["chip_every"] > 0 and self.step % p["chip_every"] == 0:
            act, chip = s["status"] == A.ACTIVE, s["status"] == A.CHIP
            off = act & (s["x"][:, 2] < pose[2] + t["tip_dz"] - 1.5 * p["dx"]) & (s["D"] > 1e-6)
            dg = s["sig"].diagonal(dim1=1, dim2=2)
            s["sres"] = torch.where(off, torch.maximum(s["sres"], torch.sqrt((dg * dg).sum(1))), s["sres"])
            s["sig"] = torch.where(off[:, None, None], 0.0, s["sig"])
            s["D"] = torch.where(off, s["D"].clamp_min(p["D_th"]), s["D"])
            s["status"] = torch.where(off, A.CHIP, s["status"])
            free = chip & (s["D"] >= 1.5 * p["D_th"])
            ident = torch.arange(lo, lo + free.numel(), device=free.device)
            h = (ident * 2654435761) & 0xFFFFFFFF
            r = torch.stack([(h >> 16) & 255, (h >> 8) & 255, h & 255], 1).double() / 255 - 0.5
            kick = r * (0.3 * s["v"].norm(dim=1) + 0.5)[:, None]
            s["v"] = torch.where(free[:, None], s["v"] + kick, s["v"])
            s["D"] = torch.where(free, 0.5 * p["D_th"], s["D"])
        if p.get("contact_every") and (self.step + 1) % p["contact_every"] == 0:
            px, pz = (t["position"][a] + t["velocity"][a] * (self.time + dt) for a in (0, 2))
            phi, nx, nz = _tool_distance(t, s["x"][:, 0], s["x"][:, 2], px, pz)
            nrm = torch.stack([nx, torch.zeros_like(nx), nz], 1)
            pen = p["contact_radius"] - phi
            hit = (pen > 0) & (s["status"] != A.INACTIVE) & (s["status"] != A.FIXED)
            vn = (s["v"] * nrm).sum(1)
            v = s["v"] - vn.clamp_max(0.0)[:, None] * nrm
            tv = v - vn[:, None] * nrm
            tvm = tv.norm(dim=1)
            m = p["particle_mass"]
            nf = torch.where(tvm > 0, (m * pen / dt ** 2).clamp_min(1e-15), torch.full_like(tvm, 1e-15))
            slide = (p["contact_friction"] * nf * dt / max(m, 1e-15) / tvm.clamp_min(1e-300)).clamp_max(1.0)
            v = v - tv * torch.where(tvm > 0, slide, 0.0)[:, None]
            warm = nf * v.norm(dim=1) * dt * (1 - p["contact_heat_partition"])
            warm = warm / (max(max(p["rho_phys"], 1.0) * max(p["particle_volume"], 1e-24), 1e-15) * p["cp"])
            s["x"] = torch.where(hit[:, None], s["x"] + nrm * pen[:, None], s["x"])
            s["v"] = torch.where(hit[:, None], v, s["v"])
            s["T"] = torch.where(hit & (warm > 0), (s["T"] + warm).clamp_max(p["Tm"]), s["T"])

    def fields(self):
        s, n = self.st, self.st["status"].numel()
        sg = s["sig"].reshape(n, 9)[:, [0, 4, 8, 1, 2, 5]]
        return dict(position=s["x"], velocity=s["v"], temperature=s["T"], F=s["F"].reshape(n, 9),
                    Fp=s["Fp"].reshape(n, 9), C=s["C"].reshape(n, 9), stress=sg, plastic_strain=s["eps"],
                    strain_rate=s["edot"], damage=s["D"], residual=s["sres"], status=s["status"].int())

    def metrics(self):
        p, s = self.p, self.st
        live = s["status"] != A.INACTIVE
        m, V = p["particle_mass"], p["particle_volume"]
        tr = s["sig"].diagonal(dim1=1, dim2=2).sum(1)
        dev = s["sig"] - (tr / 3)[:, None, None] * torch.eye(3, device=tr.device)
        vm = torch.sqrt(1.5 * (dev * dev).sum((1, 2)))
        bulk = p["E"] / (3 * (1 - 2 * p["nu"]))
        nl = int(live.sum())
        out = dict(mass=m * nl, kinetic=float(0.5 * m * (s["v"] ** 2).sum(1)[live].sum()),
                   internal_elastic=float(V * (vm ** 2 / (6 * self.mu) + (tr / 3) ** 2 / (2 * bulk))[live].sum()),
                   thermal=float(p["rho_phys"] * V * p["cp"] * (s["T"] - p["Tamb"])[live].sum()),
                   max_temperature=float(s["T"][live].max()), max_von_mises=float(vm[live].max()),
                   mean_plastic_strain=float(s["eps"][live].sum()) / max(nl, 1))
        out["momentum"] = (m * s["v"][live].sum(0)).cpu().numpy()
        out["counts"] = np.array([int((s["status"] == k).sum()) for k in (A.ACTIVE, A.CHIP, A.FIXED, A.INACTIVE)])
        return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] in ("sweep", "served"):
        ws = _sweep(case, seed)
        got = []
        for i, w in enumerate(ws):
            pos, status = _points(w, dev)
            T = torch.full_like(pos[:, 0], w["box"]["T0"])
            e = _Exact(w, dict(x=pos, v=torch.zeros_like(pos), T=T, status=status))
            e.advance(case["steps"] + (7 * (i % 4) if case["kind"] == "served" else 0), w["dt"])
            got.append((e.fields() if case["kind"] == "sweep" else None, e.metrics()))
        if case["kind"] == "sweep":
            return [{k: torch.cat([f[k] for f, _ in got]) for k in got[0][0]}, [got[0][1], got[-1][1]]]
        out = {k: np.array([m[k] for _, m in got]) for k in METRICS + ("momentum",)}
        out.update({k: np.array([m["counts"][j] for _, m in got]) for j, k in enumerate(COUNTS)})
        return out
    if case["wx"] * case["wy"] * case["wz"] * case["ppc"] * case["steps"] > 6e7:
        return None
    w = _workpiece(case)
    force = None
    if case["developed"]:
        st = _developed(w, seed, dev)
    else:
        pos, status = _points(w, dev)
        v, T, _ = _field(w, pos, seed)
        st = dict(x=pos, v=v, T=T, status=status)
    if case["kind"] == "coupling":
        force = -2e-3 * w["params"]["particle_mass"] / w["dt"] * st["v"]
        st["T"] = 0.999 * st["T"] + 1e-3 * w["params"]["Tamb"]
    e = _Exact(w, st)
    e.advance(case["steps"], w["dt"], force)
    return [e.fields(), e.metrics()]
