"""Timed cases of the tracer advection library, through its public entry points.

A program holds one library instance per process (mesh, flow, schemes on the
device); what changes from call to call are the tracer fields.  One pass of
most cases is what a coupled model does in a coupling interval: give the
library its tracers, advance them some steps, read them back.

`exact` advances the same inputs with the step written out in plain torch,
64 bits.  The mesh tables and the flow are inputs of both.
"""
import ctypes
import math

import numpy as np
import torch

from fesom2_tracer_dwarf_b200 import FESOMTracerAdvection, synth_bathymetry_smooth
from fesom2_tracer_dwarf_b200.batch import TracerBatch
from fesom2_tracer_dwarf_b200.learned import Trainer, flow, flow_amplitude, trained_params
from fesom2_tracer_dwarf_b200.workloads import cfl_dt, layered_flow_case

R_EARTH = 6367500.0
NP_OUT = {"fp64": torch.float64, "fp32": torch.float32, "bf16": torch.bfloat16}  # what a program of that precision keeps
KINDS = ("advance", "loop", "device", "io", "learned", "train", "ensemble")


def _case(kind, nx, ny, nl, steps=1, tracers=1, precision="fp64", periodic=True, hor="MUSCL", ver="PPM"):
    return {"kind": kind, "nx": nx, "ny": ny, "nl": nl, "steps": steps, "tracers": tracers, "precision": precision,
            "periodic": periodic, "hor": hor, "ver": ver, "lim": "FCT"}


def listed():
    return [
        # the reference's own analytic test case and its loop: one step, then the statistics, every step
        dict(_case("loop", 20, 20, 10, steps=10), name="dwarf_loop"),
        # a caller whose runtime owns the GPU's memory: one tracer, one step on its own device buffers
        dict(_case("device", 61, 47, 31), name="device_step"),
        # the size of FESOM's small test mesh (about 3,000 nodes, 48 levels), closed coasts
        dict(_case("advance", 58, 55, 48, steps=20, tracers=2, periodic=False), name="closed_basin"),
        # FESOM2's usual scheme pair, an odd number of tracers, a ragged closed basin
        dict(_case("advance", 241, 190, 40, steps=10, tracers=3, periodic=False, hor="MFCT", ver="QR4C"),
             name="mfct_qr4c_basin"),
        # an ordinary regional grid in double precision
        dict(_case("advance", 300, 300, 64, steps=20, tracers=2), name="fp64_300x300x64"),
        # the benchmark's grid in double precision, the drop-in mode, and in single precision
        dict(_case("advance", 1000, 1000, 64, steps=20, tracers=2), name="fp64_1000x1000x64"),
        dict(_case("advance", 1000, 1000, 64, steps=40, tracers=2, precision="fp32"), name="fp32_1000x1000x64"),
        # 16-bit tracer storage
        dict(_case("advance", 500, 500, 48, steps=20, tracers=2, precision="bf16"), name="bf16_500x500x48"),
        # one step with host I/O every step: state lives on the host
        dict(_case("io", 500, 400, 64, tracers=2), name="host_io_step"),
        # the learned antidiffusive flux: inference with the shipped network, and one training step
        dict(_case("learned", 400, 400, 32, steps=10, precision="fp32"), name="learned_400x400x32"),
        dict(_case("train", 251, 251, 32, precision="fp32"), name="train_251x251x32"),
        # an ensemble of three uneven members, eight tracers each
        dict(_case("ensemble", 233, 233, 38, steps=30, tracers=8, precision="fp32"), name="ensemble_3x8"),
    ]


def draw(rng):
    kind = rng.choice(("advance",) * 6 + KINDS[1:])
    top = {"loop": 60, "device": 75, "io": 500, "learned": 400, "train": 250, "ensemble": 230}.get(kind, 700)
    nx = int(round(math.exp(rng.uniform(math.log(17), math.log(top)))))
    ny = min(top, max(9, int(nx * rng.uniform(0.6, 1.4))))
    nl = int(round(math.exp(rng.uniform(math.log(8), math.log(48 if kind in ("device", "learned", "train") else 80)))))
    c = _case(kind, nx, ny, nl, steps=rng.randint(4, 20))
    if kind in ("io", "device", "train"):
        c["steps"] = 1
    if kind in ("learned", "train", "ensemble"):
        c["ny"] = nx
        c["precision"] = "fp32"
        c["tracers"] = 8 if kind == "ensemble" else 1
        return c
    c["periodic"] = rng.random() < 0.5
    if kind in ("advance", "io"):
        c["tracers"] = rng.randint(1, 5)
        c["hor"], c["ver"] = rng.choice((("MUSCL", "PPM"), ("MUSCL", "PPM"), ("MFCT", "QR4C"), ("UPW1", "UPW1")))
    if kind == "advance":
        c["precision"] = rng.choice(("fp64", "fp64", "fp32", "bf16"))
    return c


def _nodes(c):
    return (c["nx"] - 1) * (c["ny"] - 1) if c["periodic"] else c["nx"] * c["ny"]


def _members(c):
    """Member grids of an ensemble case: (nx, nl, periodic)."""
    return [(c["nx"], c["nl"], False), (max(12, c["nx"] * 9 // 14), c["nl"] + c["nl"] // 2, True),
            (max(9, c["nx"] * 3 // 7), max(8, c["nl"] // 2 + 2), True)]


def work(c):
    # 14 words per wet cell, tracer and step (tracer in, valuesAB in, tracer out, flow and geometry); bottom levels are
    # uniform in [3, nl]; fields cross the host boundary as 8-byte numbers once each way
    word = {"fp64": 8, "fp32": 4, "bf16": 4}[c["precision"]]
    n = _nodes(c)
    if c["kind"] == "ensemble":
        wet = sum((x - p) ** 2 * (l + 1) / 2 for x, l, p in _members(c))
        return {"bytes": c["tracers"] * (14 * word * wet * c["steps"] + 2 * 8 * wet), "flops": 300.0 * wet * c["tracers"] * c["steps"]}
    flat = c["kind"] in ("learned", "train")
    wet = n * (c["nl"] - 1 if flat else (c["nl"] + 1) / 2)
    b, f = c["tracers"] * c["steps"] * 14 * word * wet, 300.0 * wet * c["tracers"] * c["steps"]
    if flat:  # 16 -> 64 -> 64 -> 1 at every edge level, three times that with the gradient
        f += 3 * wet * c["steps"] * 2 * (16 * 64 + 64 * 64 + 64) * (3 if c["kind"] == "train" else 1)
    if c["kind"] != "device":
        b += c["tracers"] * 2 * 8 * n * (c["nl"] - 1)
    return {"bytes": b, "flops": f}


# ---- the program's library instance -----------------------------------------
class _Program:
    """The process's library instance and what is loaded in it."""

    def __init__(self):
        self.api = FESOMTracerAdvection()
        self.key = self.mesh_key = self.batch = self.trainer = self.params = None

    def close(self):
        if self.batch is not None:
            self.batch.close()
        self.batch = self.trainer = self.params = None
        self.api.cleanup()
        self.key = self.mesh_key = None

    def load(self, c):
        key = tuple(c[k] for k in ("kind", "nx", "ny", "nl", "tracers", "precision", "periodic", "hor", "ver"))
        if key == self.key:
            return
        mesh_key = (c["nx"], c["ny"], c["nl"], c["periodic"])
        if c["kind"] not in ("advance", "loop", "device", "io") or mesh_key != self.mesh_key:
            self.close()
        {"ensemble": self._ensemble, "train": self._train, "learned": self._learned}.get(c["kind"], self._grid)(c)
        self.key = key

    def _grid(self, c):
        api, mesh_key = self.api, (c["nx"], c["ny"], c["nl"], c["periodic"])
        if self.mesh_key != mesh_key:
            g = layered_flow_case(api, c["nx"], c["nl"], ny=c["ny"], periodic=c["periodic"])
            self.uv, self.w, self.dt, self.mesh_key = g.uv, g.w, g.dt, mesh_key
        api.set_precision(c["precision"])
        api.allocate_tracers(c["tracers"])
        for t in range(1, c["tracers"] + 1):
            api.set_scheme(t, c["hor"], c["ver"], c["lim"])
        api.set_velocity(self.uv, self.w)
        api.set_ab_refresh(c["kind"] != "loop")  # the reference's drivers leave valuesAB as it was set
        if c["kind"] == "device" and api.lib.tracer_init_for_advection() != 0:
            raise RuntimeError(api.lib.tracer_last_error().decode())

    def _flat(self, c):
        """The learned configuration's grid: flat bottom, depth-independent non-divergent flow."""
        api = self.api
        api.init_analytic(c["nx"], c["ny"], c["nl"], periodic=True, full_rings=True, left_oriented=True)
        self.uv, self.w = flow(api, 3, flow_amplitude(api, 3))
        self.dt = cfl_dt(api, c["nx"], c["ny"], c["nl"], self.uv, self.w)

    def _learned(self, c):
        api = self.api
        self._flat(c)
        api.set_precision("fp32")
        api.allocate_tracers(1)
        api.set_scheme(1, "MUSCL", "PPM", "FCT")
        api.set_velocity(self.uv, self.w)
        api.set_ab_refresh(True)
        self.params = trained_params()
        if api.lib.tracer_learn_set(self.params.ctypes.data_as(ctypes.c_void_p), 1) != 0:
            raise RuntimeError(api.lib.tracer_last_error().decode())

    def _train(self, c):
        self._flat(c)
        self.params = trained_params()
        self.trainer = Trainer(c["nx"], c["nl"], self.params)

    def _ensemble(self, c):
        self.batch, self.members, dts = TracerBatch(), [], []
        for m, (nx, nl, periodic) in enumerate(_members(c)):
            self.api.cleanup()
            g = layered_flow_case(self.api, nx, nl, periodic=periodic, seed=17 * m + 1)
            self.batch.add_member(nx, nx, nl, c["tracers"], periodic=periodic, node_K=g.K)
            self.batch.set_velocity(m, g.uv, g.w)
            self.members.append({"nx": nx, "nl": nl, "periodic": periodic, "K": g.K, "uv": g.uv, "w": g.w, "dt": g.dt,
                                 "shape": g.T.shape})
            dts.append(g.dt)
        self.api.cleanup()
        self.batch.configure(dts, "MUSCL", "PPM", "FCT")
        self.batch.set_path("separate")


_program = None


def _load(c):
    global _program
    if _program is None:
        _program = _Program()
    _program.load(c)
    return _program


def _field(shape, seed, kind):
    """Temperature-like noise and blobs (0), salinity-like (1), or smooth blobs and fronts (2): (nl-1, nodes)."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    L, N = shape
    if kind == 1:
        v = 35.0 + 0.5 * torch.randn(N, L, generator=g, device="cuda", dtype=torch.float64)
    else:
        x = torch.linspace(0.0, 1.0, N, device="cuda", dtype=torch.float64)[:, None]
        z = torch.linspace(0.0, 1.0, L, device="cuda", dtype=torch.float64)[None, :]
        a = torch.rand(6, generator=g, device="cuda", dtype=torch.float64).tolist()
        v = sum(2.0 * torch.exp(-((x - a[q]) / 0.05) ** 2 - ((z - a[q + 3]) / 0.3) ** 2) for q in range(3))
        v = v + (20.0 * torch.rand(N, L, generator=g, device="cuda", dtype=torch.float64) if kind == 0 else
                 10.0 + 2.0 * torch.sin(2.0 * math.pi * (40.0 * x + a[0])) * torch.cos(math.pi * z)
                 + torch.tanh(200.0 * torch.sin(2.0 * math.pi * (x * math.sqrt(N) / 9.0 + a[1]))))
    return v  # (N, L) row-major: the library's (L, N) Fortran order


def _inputs(c, seed):
    """The tracer fields of one state, on the GPU, (nodes, nl-1) each."""
    if c["kind"] == "ensemble":
        return [_field(m["shape"], seed * 1009 + 64 * i + t, t % 2) for i, m in enumerate(_load(c).members)
                for t in range(c["tracers"])]
    shape = (c["nl"] - 1, _nodes(c))
    if c["kind"] in ("learned", "train"):
        T = _field(shape, seed * 1009, 2)
        return [T, T + 0.02 * _field(shape, seed * 1009 + 1, 2)] if c["kind"] == "train" else [T]
    return [_field(shape, seed * 1009 + t, t % 2) for t in range(c["tracers"])]


class _State:
    """Page-locked host arrays of one state: the fields, and where the results go."""

    def __init__(self, c, seed):
        self.c, self.p = c, _load(c)
        self.fields = [np.asfortranarray(v.cpu().numpy().T) for v in _inputs(c, seed)]
        self.out = [np.zeros(v.shape, order="F") for v in self.fields]
        for a in self.fields + self.out:
            self.p.api.pin(a)

    def __del__(self):
        for a in getattr(self, "fields", []) + getattr(self, "out", []):
            if a.ctypes.data in self.p.api._pinned:
                self.p.api.unpin(a)


class _DeviceState:
    """Device buffers of the caller: nod2D columns of the library's level stride."""

    def __init__(self, c, seed):
        self.c, self.p = c, _load(c)
        self.T = self._columns(_inputs(c, seed)[0])
        self.out = torch.zeros_like(self.T)
        torch.cuda.synchronize()

    def _columns(self, v):
        col = torch.zeros(v.shape[0], self.p.api.mesh_dims()["level_stride"], dtype=torch.float64, device="cuda")
        col[:, : v.shape[1]] = v
        return col


def prepare(c, seed):
    return (_DeviceState if c["kind"] == "device" else _State)(c, seed)


def _read(s):
    """The results as the program keeps them, in its precision."""
    api, shape = s.p.api, s.out[0].shape
    for t, a in enumerate(s.out, 1):
        if api.lib.tracer_get_values_id(t, a.ctypes.data_as(ctypes.c_void_p), shape[0], shape[1]) != 0:
            raise RuntimeError(api.lib.tracer_last_error().decode())
    return [torch.from_numpy(a.T).to(NP_OUT[s.c["precision"]]) for a in s.out]


def run(s):
    c, p = s.c, s.p
    api = p.api
    if c["kind"] == "device":
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        if api.lib.tracer_advect_device_noalloc(1, ptr(s.T), ptr(s.T), ptr(s.out), p.dt) != 0:
            raise RuntimeError(api.lib.tracer_last_error().decode())
        return s.out
    if c["kind"] == "io":
        api.advect_step_io(p.dt, s.fields, s.out)
        return s.out
    if c["kind"] == "ensemble":
        b = p.batch
        at = [(m, t) for m in range(len(p.members)) for t in range(1, c["tracers"] + 1)]
        for (m, t), v in zip(at, s.fields):
            b.set_values(m, t, v)
        b.steps(c["steps"], graph=True)
        for (m, t), a in zip(at, s.out):
            if b.lib.tracer_batch_get_values(m, t, a.ctypes.data_as(ctypes.c_void_p)) != 0:
                raise RuntimeError(b.lib.tracer_last_error().decode())
        return [torch.from_numpy(a.T).to(torch.float32) for a in s.out]
    if c["kind"] == "train":
        tr = p.trainer
        tr.load(p.params, on=False)
        loss = tr.step_loss({"seed": 0, "uv": p.uv, "w": p.w, "dt": p.dt, "snaps": s.fields}, 0, lr=1e-4, update=True)
        grad = np.zeros_like(p.params)
        if tr.lib.tracer_learn_grad(grad.ctypes.data_as(ctypes.c_void_p)) != 0:
            raise RuntimeError(tr.lib.tracer_last_error().decode())
        return {"loss": loss, "gradient": grad}
    for t, v in enumerate(s.fields, 1):
        api.set_values(t, v)
    if c["kind"] == "loop":
        stats = []
        for _ in range(c["steps"]):
            if api.advect_step(p.dt) != 0:
                raise RuntimeError(api.lib.tracer_last_error().decode())
            q = api.get_statistics(1)
            stats.append([q["min"], q["max"], q["sum"]])
        return {"values": _read(s), "statistics": np.array(stats)}
    api.advect_steps(c["steps"], p.dt)
    return _read(s)


# ---- the step in 64 bits ------------------------------------------------------
def _mesh(api, uv, w):
    d = api.mesh_dims()
    nl, N, T, E = d["nl"], d["nod2D"], d["elem2D"], d["edge2D"]

    def arr(name, *shape):
        a = torch.from_numpy(api.mesh_array(name)).cuda().reshape(shape)
        return a.long() if a.dtype == torch.int32 else a

    m = {"L": nl - 1, "N": N, "E": E, "en": arr("elem2D_nodes", T, 3) - 1, "ed": arr("edges", E, 2) - 1,
         "tri": arr("edge_tri", E, 2) - 1, "nle": arr("nlevels", T) - 1, "nln": arr("nlevels_nod2D", N) - 1,
         "nlmin": arr("nlevels_nod2D_min", N), "ud": arr("edge_up_dn_tri", E, 2) - 1, "nbl": arr("nboundary_lay", N),
         "earea": arr("elem_area", T), "area": arr("area", N, nl), "asv": arr("areasvol", N, nl)[:, : nl - 1],
         "dxdy": arr("edge_dxdy", E, 2), "cross": arr("edge_cross_dxdy", E, 4), "gs": arr("gradient_sca", T, 6),
         "h": arr("hnode", N, nl - 1), "hn": arr("hnode_new", N, nl - 1), "helem": arr("helem", T, nl - 1),
         "zbar": arr("zbar", nl), "W": torch.from_numpy(w.T).cuda()}
    k = torch.arange(nl - 1, device="cuda")[None]
    m["wet"], m["wete"] = k < m["nln"][:, None], k < m["nle"][:, None]
    m["asv"] = torch.where(m["wet"], m["asv"], torch.ones((), dtype=torch.float64, device="cuda"))
    u = torch.from_numpy(uv.T).cuda()  # (T, L, 2)
    vf = torch.zeros(E, nl - 1, dtype=torch.float64, device="cuda")
    edge_levels = torch.zeros(E, dtype=torch.long, device="cuda")
    for s, sign in ((0, 1.0), (1, -1.0)):
        t = m["tri"][:, s]
        has, t = t >= 0, t.clamp(min=0)
        dx, dy = m["cross"][:, 2 * s, None], m["cross"][:, 2 * s + 1, None]
        f = sign * (u[t, :, 0] * dy - u[t, :, 1] * dx) * m["helem"][t]
        vf += torch.where(has[:, None] & m["wete"][t], f, torch.zeros_like(f))
        edge_levels = torch.maximum(edge_levels, torch.where(has, m["nle"][t], torch.zeros_like(t)))
    m["vf"], m["wetd"] = vf, k < edge_levels[:, None]
    return m


def _mlp(f, p):
    gelu = lambda z: 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))  # noqa: E731
    h = gelu(f @ p[:1024].reshape(64, 16).T + p[1024:1088])
    h = gelu(h @ p[1088:5184].reshape(64, 64).T + p[5184:5248])
    return h @ p[5248:5312] + p[5312]


def _edge_flux(m, T, AB, dt, hor, net):
    """Upwind flux of T and antidiffusive flux (high order of AB minus it) of every edge level, positive into node 1."""
    L, vf = m["L"], m["vf"]
    n1, n2 = m["ed"].T
    up = lambda t: -0.5 * (t[n1] * (vf + vf.abs()) + t[n2] * (vf - vf.abs()))  # noqa: E731
    lo = torch.where(m["wetd"], up(T), torch.zeros_like(vf))
    if hor == "UPW1":
        return lo, torch.where(m["wetd"], up(AB), torch.zeros_like(vf)) - lo
    k = torch.arange(L, device="cuda")[None]
    a = m["earea"][:, None] * m["wete"]
    vol = torch.zeros(m["N"], L, dtype=T.dtype, device="cuda")
    for q in range(3):
        vol.index_add_(0, m["en"][:, q], a)
    u, d = m["ud"].T
    shared = (u >= 0)[:, None] & (d >= 0)[:, None] & (k + 1 <= torch.minimum(m["nlmin"][n1], m["nlmin"][n2])[:, None] - 1)
    gu, gd = [], []
    for x in range(2):
        g = sum(m["gs"][:, 3 * x + q, None] * AB[m["en"][:, q]] for q in range(3))
        r = torch.zeros(m["N"], L, dtype=T.dtype, device="cuda")
        for q in range(3):
            r.index_add_(0, m["en"][:, q], g * a)
        r = r / vol
        gu.append(torch.where(shared, g[u.clamp(min=0)], r[n1]))
        gd.append(torch.where(shared, g[d.clamp(min=0)], r[n2]))
        del g, r
    t1, t2 = AB[n1], AB[n2]
    ex, ey = m["dxdy"][:, 0, None] * R_EARTH, m["dxdy"][:, 1, None] * R_EARTH
    x2 = 2.0 * (t2 - t1) + ex * gd[0] + ey * gd[1]
    x1 = 2.0 * (t2 - t1) + ex * gu[0] + ey * gu[1]
    c1, c2 = ((m["nbl"][n][:, None] - (k + 1) >= 0).to(T.dtype) if hor == "MUSCL" else torch.ones_like(vf) for n in (n1, n2))
    m2, m1 = t2 - x2 / 6.0 * c2, t1 + x1 / 6.0 * c1
    ho = -vf * 0.5 * (m1 + m2)  # ph = 1
    adf = torch.where(m["wetd"], ho, torch.zeros_like(ho)) - lo
    if net is not None:
        fwd = vf >= 0
        pick = lambda a, b: torch.where(fwd, a, b)  # noqa: E731
        tu, td, xu, xd = pick(t1, t2), pick(t2, t1), pick(x1, -x2), pick(x2, -x1)
        sig = (td - tu).abs() + (xu.abs() + xd.abs()) / 6.0 + 1e-6 * (tu.abs() + td.abs()) + 1e-20
        vcell = m["asv"] * m["hn"]
        cour = (vf.abs() * dt / pick(vcell[n1], vcell[n2])).clamp(max=4.0)
        trans = (-ey * pick(gu[0], gd[0]) + ex * pick(gu[1], gd[1])) / sig
        f0, f1, f2 = (td - tu) / sig, xu / 6.0 / sig, xd / 6.0 / sig
        level = (k / max(1, L - 1)).to(T.dtype).expand_as(vf)
        feats = [f0, f1, f2, (0.5 * (m1 + m2) - tu) / sig, cour, cour * cour, pick(c1, c2), pick(c2, c1), level,
                 shared.to(T.dtype), f0.abs(), f1 - f2, torch.where(xu * xd > 0, 1.0, -1.0),
                 torch.minimum(f1.abs(), f2.abs()), trans.clamp(-8.0, 8.0), torch.ones_like(vf)]
        f = torch.stack(feats, -1)
        y = _mlp(f, net) if net.requires_grad else torch.cat([_mlp(b, net) for b in f.split(20000)])
        adf = adf - vf * sig * y
    return lo, adf


def _vertical(m, T, AB, dt, ver):
    """Upwind flux of T and antidiffusive flux at every interface, (N, L+1), positive upwards out of the layer above."""
    L, N, W, A, nln = m["L"], m["N"], m["W"], m["area"], m["nln"][:, None]
    i = torch.arange(L + 1, device="cuda")[None]
    z1 = torch.zeros(N, 1, dtype=T.dtype, device="cuda")
    above = lambda v: torch.cat([z1, v], 1)  # noqa: E731  value in the layer above the interface
    below = lambda v: torch.cat([v, z1], 1)  # noqa: E731
    top, bottom = i == 0, i >= nln

    def upwind(v):
        f = -(0.5 * (below(v) * (W + W.abs()) + above(v) * (W - W.abs())) * A)
        f = torch.where(top, -(W * below(v) * A), f)
        return torch.where(bottom, torch.zeros_like(f), f)

    lo = upwind(T)
    if ver == "UPW1":
        return lo, upwind(AB) - lo
    if ver == "QR4C":  # pv = 1
        Z = 0.5 * (m["zbar"][:-1] + m["zbar"][1:])
        g = (AB[:, :-1] - AB[:, 1:]) / (Z[:-1] - Z[1:])[None]  # at interface 1 .. L-1
        qc = torch.cat([z1, g, z1], 1)
        qu, qd = torch.cat([qc[:, 1:], z1], 1), torch.cat([z1, qc[:, :-1]], 1)
        zb, zc, za = m["zbar"][None], torch.cat([Z, Z[-1:]])[None], torch.cat([Z[:1], Z])[None]
        v1 = below(AB) + (2.0 * qc + qu) * (zb - zc) / 3.0
        v2 = above(AB) + (2.0 * qc + qd) * (zb - za) / 3.0
        f = -(0.5 * (v1 + v2)) * W * A
        f = torch.where((i == 1) | (i == nln - 1), -(0.5 * (above(AB) + below(AB)) * W * A), f)
        f = torch.where(top, -(below(AB) * W * A), f)
        f = torch.where(bottom, torch.zeros_like(f), f)
        # a two-layer column: its one inner interface is assigned twice, the second time minus the first
        return lo, torch.where((i == 1) & (nln == 2), lo, f - lo)
    # PPM
    hn = m["hn"]
    at = lambda v, s: torch.roll(v, -s, 1)  # noqa: E731  value s layers further down
    k = i[:, :L]
    up_, dn_ = AB - at(AB, -1), at(AB, 1) - AB
    hm, hp, hp2 = at(hn, -1), at(hn, 1), at(hn, 2)
    s = hn / (hm + hn + hp) * ((2.0 * hm + hn) / (hp + hn) * dn_ + (hn + 2.0 * hp) / (hm + hn) * up_)
    s = torch.where(dn_ * up_ > 0, torch.copysign(torch.minimum(s.abs(), 2.0 * torch.minimum(dn_.abs(), up_.abs())), s),
                    torch.zeros_like(s))
    s = torch.where((k >= 1) & (k <= nln - 2), s, torch.zeros_like(s))
    h0, h1, hm1, h2 = at(hn, -1), hn, at(hn, -2), at(hn, 1)  # interface k: layers k-1, k, k-2, k+1
    cc = 2.0 * h1 * h0 / (h0 + h1) * ((hm1 + h0) / (2.0 * h0 + h1) - (h2 + h1) / (2.0 * h1 + h0))
    tv = at(AB, -1) + h0 / (h0 + h1) * up_ + (cc * up_ - h0 * (hm1 + h0) / (2.0 * h0 + h1) * s
                                              + h1 * (h1 + h2) / (h0 + 2.0 * h1) * at(s, -1)) / (hm1 + h0 + h1 + h2)
    tv = torch.where(k == 1, 0.5 * (at(AB, -1) + AB), tv)
    tv = torch.where(k == nln - 1, torch.where(torch.signbit(W[:, :L]), at(AB, -1), AB), tv)
    tv = torch.where(k == 0, AB, tv)
    aL, aR = tv, torch.where(k == nln - 1, AB, at(tv, 1))
    flat = (aR - AB) * (AB - aL) <= 0
    aL, aR = torch.where(flat, AB, aL), torch.where(flat, AB, aR)
    aL = torch.where((aR - aL) * (AB - 0.5 * (aL + aR)) > (aR - aL) ** 2 / 6.0, 3.0 * AB - 2.0 * aR, aL)
    aR = torch.where((aR - aL) * (AB - 0.5 * (aL + aR)) < -((aR - aL) ** 2) / 6.0, 3.0 * AB - 2.0 * aL, aR)
    aj = 6.0 * (AB - 0.5 * (aL + aR))
    one = torch.ones((), dtype=T.dtype, device="cuda")
    x = torch.minimum(below(1.0 / m["h"]) * W * dt, one)
    dn = -below(aL) - 0.5 * x * (below(aR - aL) + (1.0 - 2.0 / 3.0 * x) * below(aj))
    x = torch.minimum(-above(1.0 / m["h"]) * W * dt, one)
    upw = -above(aR) + 0.5 * x * (above(aR - aL) - (1.0 - 2.0 / 3.0 * x) * above(aj))
    f = torch.where(W > 0, dn, torch.where(W < 0, upw, torch.zeros_like(dn))) * A * W
    f = torch.where(top, -(below(tv) * W * A), f)
    return lo, torch.where(bottom, torch.zeros_like(f), f) - lo


def _step(m, T, AB, dt, hor, ver, net=None):
    """One step of one tracer with the FCT limiter."""
    n1, n2 = m["ed"].T
    wet, nln = m["wet"], m["nln"][:, None]
    k = torch.arange(m["L"], device="cuda")[None]
    zero = torch.zeros((), dtype=T.dtype, device="cuda")
    flo, adf = _edge_flux(m, T, AB, dt, hor, net)
    vlo, adv = _vertical(m, T, AB, dt, ver)
    into = lambda f1, f2: torch.zeros_like(T).index_add(0, n1, f1).index_add(0, n2, f2)  # noqa: E731
    lo = (T * m["h"] + (into(flo, -flo) + vlo[:, :-1] - vlo[:, 1:]) * dt / m["asv"]) / m["hn"]
    lo = torch.where(wet, lo, zero)

    def cluster(v, sign):  # the largest of sign * v over the elements around each node, then over the layers next to it
        e = torch.stack([(sign * v)[m["en"][:, q]] for q in range(3)]).amax(0)
        e = torch.where(m["wete"], e, torch.full_like(zero, -1e3))
        b = torch.full_like(T, -math.inf)
        for q in range(3):
            b.scatter_reduce_(0, m["en"][:, q, None].expand_as(e), e, "amax")
        inner = torch.stack([torch.roll(b, 1, 1), b, torch.roll(b, -1, 1)]).amax(0)
        return sign * torch.where((k == 0) | (k == nln - 1), b, inner)

    bmax = cluster(torch.maximum(lo, T), 1.0) - lo
    bmin = cluster(torch.minimum(lo, T), -1.0) - lo
    pos, neg = (lambda f: f.clamp(min=0.0)), (lambda f: f.clamp(max=0.0))
    fp = pos(adv[:, :-1]) + pos(-adv[:, 1:]) + into(pos(adf), pos(-adf))
    fm = neg(adv[:, :-1]) + neg(-adv[:, 1:]) + into(neg(adf), neg(-adf))
    one = torch.ones_like(zero)
    rp = torch.minimum(one, bmax / (fp * dt / m["asv"] + 1e-16))
    rm = torch.minimum(one, bmin / (fm * dt / m["asv"] - 1e-16))
    f = adf * torch.where(adf >= 0, torch.minimum(rp[n1], rm[n2]), torch.minimum(rm[n1], rp[n2]))
    z1 = torch.ones(T.shape[0], 1, dtype=T.dtype, device="cuda")
    above, below = (lambda r: torch.cat([z1, r], 1)), (lambda r: torch.cat([r, z1], 1))
    ae = torch.where(adv >= 0, torch.minimum(above(rm), below(rp)), torch.minimum(above(rp), below(rm)))
    i = torch.arange(m["L"] + 1, device="cuda")[None]
    fv = torch.where(i < nln, ae * adv, zero)
    new = lo + (T * (m["hn"] - m["h"]) + (into(f, -f) + fv[:, :-1] - fv[:, 1:]) * dt / m["asv"]) / m["hn"]
    return torch.where(wet, new, T)


def exact(c, seed):
    p = _load(c)
    fields, api = _inputs(c, seed), p.api
    with torch.no_grad():
        if c["kind"] == "ensemble":
            out = []
            for i, q in enumerate(p.members):
                api.cleanup()
                api.init_analytic(q["nx"], q["nx"], q["nl"], periodic=q["periodic"], node_K=q["K"], left_oriented=True)
                m = _mesh(api, q["uv"], q["w"])
                for T in fields[i * c["tracers"]:(i + 1) * c["tracers"]]:
                    for _ in range(c["steps"]):
                        T = _step(m, T, T, q["dt"], "MUSCL", "PPM")
                    out.append(T)
            api.cleanup()
            return out
        m = _mesh(api, p.uv, p.w)
    if c["kind"] == "train":
        net = torch.from_numpy(p.params).cuda().double().requires_grad_(True)
        T, target = fields
        new = _step(m, T, T, p.dt, "MUSCL", "PPM", net)
        vol = m["asv"] * m["hn"] * m["wet"]
        loss = (vol * (new - target) ** 2).sum() / vol.sum()
        loss.backward()
        return {"loss": float(loss.detach()), "gradient": net.grad}
    with torch.no_grad():
        net = None if p.params is None else torch.from_numpy(p.params).cuda().double()
        out, stats = [], []
        for T in fields:
            AB = T
            for _ in range(c["steps"]):
                T = _step(m, T, AB if c["kind"] == "loop" else T, p.dt, c["hor"], c["ver"], net)
                stats.append(torch.stack([T.min(), T.max(), T.sum()]))
            out.append(T)
        if c["kind"] == "device":
            col = torch.zeros(T.shape[0], api.mesh_dims()["level_stride"], dtype=torch.float64, device="cuda")
            col[:, : T.shape[1]] = torch.where(m["wet"], T, torch.zeros_like(T))
            return col
        if c["kind"] == "loop":
            return {"values": out, "statistics": torch.stack(stats)}
        return [T.T for T in out] if c["kind"] == "io" else out
