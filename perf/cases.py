"""The work that programs have this library do, as cases that can be timed.

Every case goes through the public Python mirror of the C interface
(astaroth_b200.Device and Ensemble). A stepping case is what a program does that
keeps its fields in GPU arrays of its own: load them, advance a number of steps,
fill the ghost zones and store the fields again. `kind` says how the steps are
made:

  steps        acDeviceIntegrateSteps: whole steps of a fixed time step
  cfl          acDeviceIntegrateStepsCFL: the time step follows the state
  substeps     the reference's own loop: ghost fill, substep, buffer swap
  walls        the same with symmetric or antisymmetric walls
               (acDeviceGeneralBoundconds)
  forced       every step a new helical forcing and the four diagnostics that the
               standalone sample prints, folded into the step
  diagnostics  every step followed by MAX, MIN and RMS of |u| and of every field
               and by rms_exp of lnrho, 28 values read back
  snapshot     pinned host memory in and out, max |u| read back every step
  ensemble     independent meshes of uneven sizes advanced together; their state
               stays with the library, and every pass stores it

`flavour` is the library: sp (FP32), dp (FP64) or mixed (FP32 stencils on a
compensated state).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from astaroth_b200 import abi
from astaroth_b200.device import Device, Ensemble

NG = 3
LNRHO, UX, UY, UZ, AX, AY, AZ, SS = range(8)
# configuration of the library's own benchmark; every other parameter keeps the
# reference's default configuration
PHYS = dict(gamma=5.0 / 3.0, nu_visc=5e-3, eta=5e-3, cs_sound=1.0, cp_sound=1.0)
ZETA, MU0, LNT0, LNRHO0 = 0.01, 1.4, 1.2, 1.3
CDT, CDTV = 0.4, 0.3
DT = 1e-3
# ensemble: per-member viscosity and resistivity, log-uniform
NU_RANGE = (1e-3, 1e-2)


def listed():
    return [
        # the smallest mesh in use: an ensemble member's size on its own; six
        # kernels a step, each a few microseconds
        dict(name="sp_32_steps", kind="steps", flavour="sp", nx=32, ny=32, nz=32, steps=20),
        # the reference's default configuration (64^3), its loop with the time
        # step chosen from the state
        dict(name="sp_64_cfl", kind="cfl", flavour="sp", nx=64, ny=64, nz=64, steps=20),
        # a small double-precision run, sizes that fill no tile, the reference's
        # substep loop
        dict(name="dp_ragged_substeps", kind="substeps", flavour="dp", nx=61, ny=70, nz=53,
             steps=10),
        # an ordinary single-precision run on a ragged mesh
        dict(name="sp_ragged_substeps", kind="substeps", flavour="sp", nx=157, ny=131, nz=118,
             steps=10),
        # closed box: the general boundary conditions of acIntegrateGBC
        dict(name="sp_128_walls", kind="walls", flavour="sp", nx=128, ny=128, nz=128, steps=6,
             wall=1),
        # forced turbulence in mixed precision with the standalone's diagnostics
        dict(name="mixed_192_forced", kind="forced", flavour="mixed", nx=192, ny=192, nz=192,
             steps=6),
        # the 256^3 workload with the standalone's full diagnostics print
        dict(name="sp_256_diagnostics", kind="diagnostics", flavour="sp", nx=256, ny=256, nz=256,
             steps=2),
        # a program whose fields live in host memory
        dict(name="sp_192_snapshot", kind="snapshot", flavour="sp", nx=192, ny=192, nz=192,
             steps=4),
        # parameter sweep: 64 meshes of 32^3 ... 128^3
        dict(name="sp_ensemble_64", kind="ensemble", flavour="sp", members=64, nmin=32, nmax=128,
             steps=4),
        # the 256^3 double-precision workload
        dict(name="dp_256_steps", kind="steps", flavour="dp", nx=256, ny=256, nz=256, steps=6),
        # the reference's benchmark size in single precision
        dict(name="sp_512_steps", kind="steps", flavour="sp", nx=512, ny=512, nz=512, steps=8),
        # the benchmark's headline: 512^3 in mixed precision
        dict(name="mixed_512_steps", kind="steps", flavour="mixed", nx=512, ny=512, nz=512,
             steps=8),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], half of them odd or ragged."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 0.5 else max(lo, n // 8 * 8)


def draw(rng):
    kind = rng.choice(["steps", "steps", "cfl", "substeps", "walls", "forced", "diagnostics",
                       "snapshot", "ensemble"])
    flavour = rng.choice(["sp", "mixed", "dp"])
    if kind == "ensemble":
        nmin = _size(rng, 16, 48)
        return dict(kind=kind, flavour=flavour, members=rng.randrange(3, 65), nmin=nmin,
                    nmax=rng.randrange(nmin + 16, 129), steps=rng.randrange(1, 4))
    hi = {"steps": 400, "snapshot": 224, "diagnostics": 288, "walls": 192}.get(kind, 256)
    if flavour == "dp":
        hi = min(hi, 256)
    n = [_size(rng, 16, hi) for _ in range(3)]
    if rng.random() < 0.4:
        n = [n[0]] * 3
    case = dict(kind=kind, flavour=flavour, nx=n[0], ny=n[1], nz=n[2], steps=rng.randrange(2, 8))
    if kind == "walls":
        case["wall"] = rng.choice([1, 2])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _real(flavour):
    return (torch.float64, np.float64) if flavour == "dp" else (torch.float32, np.float32)


def _spacings(n):
    """A 2 pi box along every axis (so the spacing differs on uneven meshes)."""
    return [2.0 * math.pi / m for m in n]


def _fields(n, seed, member=0):
    """The eight interior fields in float64 on the GPU, indexed [z, y, x]: three
    Fourier modes of random direction and phase (|k| <= 3) and grid-scale noise."""
    nx, ny, nz = n
    rng = np.random.default_rng([seed, member])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 40)))
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") * (2.0 * math.pi / m)
          for m in (nx, ny, nz)]
    amplitude = [0.05] + [0.1] * 3 + [0.1] * 3 + [0.05]
    out = []
    for w in range(8):
        f = torch.rand((nz, ny, nx), generator=gen, dtype=torch.float32, device="cuda").double()
        f.mul_(2e-3).sub_(1e-3)
        for _ in range(3):
            k = rng.integers(-3, 4, 3)
            ph = rng.uniform(0.0, 2.0 * math.pi)
            a = amplitude[w] / 3.0
            xy = float(k[0]) * ax[0][None, :] + float(k[1]) * ax[1][:, None] + ph
            z = float(k[2]) * ax[2][:, None, None]
            f.addcmul_(torch.cos(z), a * torch.cos(xy)[None])
            f.addcmul_(torch.sin(z), -a * torch.sin(xy)[None])
        out.append(f)
    return out


def _pad(f, wall=0):
    """The field with its ghost zone: periodic, or mirrored about the walls
    (1 symmetric, 2 antisymmetric)."""
    if not wall:
        for d in (0, 1, 2):
            f = torch.cat((f.narrow(d, f.shape[d] - NG, NG), f, f.narrow(d, 0, NG)), d)
        return f
    g = torch.nn.functional.pad(f[None, None], (NG,) * 6, mode="reflect")[0, 0]
    if wall == 2:
        g = -g
        g[NG:-NG, NG:-NG, NG:-NG] = f
    return g


def _info(flavour, n, **more):
    ds = _spacings(n)
    return abi.make_info(abi.PRECISIONS[flavour], *n, dsx=ds[0], dsy=ds[1], dsz=ds[2], **PHYS,
                         **more)


def _mesh(flavour, info, tensors):
    """An AcMesh over contiguous tensors, in GPU or pinned host memory."""
    prec = abi.PRECISIONS[flavour]
    mesh = abi.mesh_type(prec)()
    mesh.info = info
    for w, t in enumerate(tensors):
        mesh.vertex_buffer[w] = C.cast(C.c_void_p(t.data_ptr()), C.POINTER(prec.real))
    return mesh


def _forcings(case, seed):
    """One forcing per step: an integer wavevector, a phase and a helical
    amplitude, as the standalone's generator draws them."""
    rng = np.random.default_rng([seed, 7])
    out = []
    for _ in range(case["steps"]):
        k = np.zeros(3)
        while not 1.0 <= np.dot(k, k) <= 9.0:
            k = rng.integers(-3, 4, 3).astype(float)
        e = np.cross(k, rng.normal(size=3))
        e /= np.linalg.norm(e)
        out.append(dict(k=k, re=e, im=np.cross(k, e) / np.linalg.norm(k),
                        phase=float(rng.uniform(-math.pi, math.pi)), magnitude=0.05, kaver=2.0))
    return out


def _members(case, seed):
    rng = np.random.default_rng([seed, 11])
    sizes = np.linspace(case["nmin"], case["nmax"], 4).round().astype(int)
    lo, hi = np.log(NU_RANGE)
    return [dict(n=[int(sizes[i % 4])] * 3, nu=float(np.exp(rng.uniform(lo, hi))),
                 eta=float(np.exp(rng.uniform(lo, hi)))) for i in range(case["members"])]


def _n(case):
    return [case["nx"], case["ny"], case["nz"]]


class State:
    """What a program has in hand: its arrays and the library's handle."""

    def __init__(self, case, seed):
        self.case = case
        self.handle = None
        flavour = case["flavour"]
        real = _real(flavour)[0]
        if case["kind"] == "ensemble":
            self.members = _members(case, seed)
            infos = [abi.make_info(abi.PRECISIONS[flavour], *m["n"],
                                   **dict(zip(("dsx", "dsy", "dsz"), _spacings(m["n"]))),
                                   **dict(PHYS, nu_visc=m["nu"], eta=m["eta"]))
                     for m in self.members]
            # one array of [member, field, z, y, x] for the members of each size
            groups = {}
            for i, m in enumerate(self.members):
                groups.setdefault(m["n"][0], []).append(i)
            self.out, self.meshes = {}, [None] * len(infos)
            for k, group in groups.items():
                side = k + 2 * NG
                self.out[k] = torch.empty((len(group), 8, side, side, side), dtype=real,
                                          device="cuda")
                for i, t in zip(group, self.out[k]):
                    for w, f in enumerate(_fields(self.members[i]["n"], seed, i)):
                        t[w].copy_(_pad(f))
                    self.meshes[i] = _mesh(flavour, infos[i], t)
            self.handle = Ensemble(flavour, infos)
            torch.cuda.synchronize()
            for i, mesh in enumerate(self.meshes):
                _ok(self.handle.lib.acEnsembleLoadMember(self.handle.handle, i, mesh))
            return
        n = _n(case)
        more = {}
        if case["kind"] == "walls":
            more = {f"bc_type_{side}_{axis}": case["wall"] for side in ("top", "bot")
                    for axis in "xyz"}
        if case["kind"] == "cfl":
            more = dict(cdt=CDT, cdtv=CDTV, dsmin=min(_spacings(n)))
        self.info = _info(flavour, n, **more)
        wall = case.get("wall", 0)
        self.fields = [_pad(f, wall).to(real) for f in _fields(n, seed)]
        if case["kind"] == "snapshot":
            self.fields = [f.cpu().pin_memory() for f in self.fields]
        self.out = [torch.empty_like(f, pin_memory=f.is_pinned()) for f in self.fields]
        self.mesh_in = _mesh(flavour, self.info, self.fields)
        self.mesh_out = _mesh(flavour, self.info, self.out)
        if case["kind"] == "forced":
            self.forcings = [_forcing_params(flavour, f) for f in _forcings(case, seed)]
        self.handle = Device(flavour, self.info)
        if case["kind"] == "forced":
            self.handle.set_forcing(True)
            self.handle.set_step_diagnostics(True)
        torch.cuda.synchronize()

    def __del__(self):
        if self.handle is not None:
            self.handle.destroy()


def _forcing_params(flavour, f):
    p = abi.forcing_type(abi.PRECISIONS[flavour])()
    p.magnitude, p.phase, p.kaver = f["magnitude"], f["phase"], f["kaver"]
    for c in range(3):
        p.k_force[c], p.ff_hel_re[c], p.ff_hel_im[c] = f["k"][c], f["re"][c], f["im"][c]
    return p


def prepare(case, seed):
    return State(case, seed)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ok(rc):
    if rc != abi.AC_SUCCESS:
        raise RuntimeError("the library returned AC_FAILURE")


def _print_values(dev):
    """MAX, MIN and RMS of |u| and of every field, as the standalone prints them,
    and its rms_exp of lnrho (raw sums for RMS, as the Device layer returns)."""
    u = (abi.VTXBUF_UUX, abi.VTXBUF_UUY, abi.VTXBUF_UUZ)
    kinds = (abi.RTYPE_MAX, abi.RTYPE_MIN, abi.RTYPE_RMS)
    values = [dev.reduce_vec_double(r, *u) for r in kinds]
    for w in range(abi.NUM_VTXBUF_HANDLES):
        values += [dev.reduce_scal_double(r, w) for r in kinds]
    return values + [dev.reduce_scal_double(abi.RTYPE_RMS_EXP, abi.VTXBUF_LNRHO)]


def run(state):
    case, dev = state.case, state.handle
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        dev.integrate_steps(DT, steps)
        for i, mesh in enumerate(state.meshes):
            _ok(dev.lib.acEnsembleStoreMember(dev.handle, i, C.byref(mesh)))
        # the ensemble fills no ghost zones for its caller: the interiors
        return [t[..., NG:-NG, NG:-NG, NG:-NG] for t in state.out.values()]
    u = (abi.VTXBUF_UUX, abi.VTXBUF_UUY, abi.VTXBUF_UUZ)
    values = []
    _ok(dev.lib.acDeviceLoadMesh(dev.handle, 0, state.mesh_in))
    if kind == "steps":
        dev.integrate_steps(DT, steps)
    elif kind == "cfl":
        dev.integrate_steps_cfl(steps)
    elif kind == "substeps":
        for _ in range(steps):
            for s in range(3):
                dev.periodic_boundconds()
                dev.integrate_substep(s, DT)
                dev.swap_buffers()
    elif kind == "walls":
        lo, hi = dev.full_box()
        outside = abi.int3(-1, -1, -1)
        for _ in range(steps):
            for s in range(3):
                _ok(dev.lib.acDeviceGeneralBoundconds(dev.handle, 0, lo, hi, state.info, outside))
                dev.integrate_substep(s, DT)
                dev.swap_buffers()
    elif kind == "forced":
        for forcing in state.forcings:
            dev.load_forcing_params(forcing)
            dev.integrate_step(DT)
            values.append([dev.reduce_vec_double(r, *u)
                           for r in (abi.RTYPE_MAX, abi.RTYPE_MIN, abi.RTYPE_RMS)] +
                          [dev.reduce_scal_double(abi.RTYPE_RMS_EXP, abi.VTXBUF_LNRHO)])
    elif kind == "diagnostics":
        for _ in range(steps):
            dev.integrate_step(DT)
            values.append(_print_values(dev))
    elif kind == "snapshot":
        for _ in range(steps):
            dev.integrate_step(DT)
            values.append([dev.reduce_vec(abi.RTYPE_MAX, *u)])
    if kind == "walls":
        _ok(dev.lib.acDeviceGeneralBoundconds(dev.handle, 0, lo, hi, state.info, outside))
    else:
        dev.periodic_boundconds()
    _ok(dev.lib.acDeviceStoreMesh(dev.handle, 0, C.byref(state.mesh_out)))
    if kind == "snapshot":
        dev.synchronize(0)  # the fields are read on the host now
    if values:
        return dict(fields=state.out, values=np.array(values, dtype=np.float64))
    return dict(fields=state.out)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Operations of one vertex and substep: 21 first derivatives (8 each), 24 second
# (10), 12 diagonal cross derivatives (14), about 250 for the right-hand sides
# and 4 per field for the update.
FLOPS = 21 * 8 + 24 * 10 + 12 * 14 + 250 + 8 * 4


def work(case):
    # bytes of a state value: the mixed state is a float and a bfloat16
    state = {"sp": 4, "mixed": 6, "dp": 8}[case["flavour"]]
    value = 8 if case["flavour"] == "dp" else 4
    meshes = ([m["n"] for m in _members(case, 0)] if case["kind"] == "ensemble" else [_n(case)])
    bytes_, flops = 0, 0
    for n in meshes:
        cells, padded = math.prod(n), math.prod(m + 2 * NG for m in n)
        # a substep reads the state and (but the first) the previous one and writes the next
        bytes_ += case["steps"] * 8 * cells * 8 * state
        flops += case["steps"] * 3 * cells * FLOPS
        # ghost zones: written and their sources read, before each substep
        bytes_ += case["steps"] * 3 * 2 * 8 * (padded - cells) * value
        # load and store: read once and written once each; the ensemble stores only
        bytes_ += (2 if case["kind"] == "ensemble" else 4) * 8 * padded * value
        if case["kind"] == "diagnostics":
            bytes_ += case["steps"] * 8 * cells * state
        if case["kind"] == "snapshot":
            bytes_ += case["steps"] * 3 * cells * state
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # Four times the relative 2-norm error against 64 bits that was measured
    # (fields stored as floats: FP32 2.2e-7, and on fine meshes 4e-7 a step at 512,
    # where its second differences cancel terms of 2.7 f / ds^2, so with n^2;
    # mixed 1.2e-7; FP64 1.4e-15 between two correct evaluations).
    if case["flavour"] == "sp":
        n = case["nmax"] if case["kind"] == "ensemble" else max(_n(case))
        return {"rel": 1e-6 + 1.6e-6 * case["steps"] * (n / 512.0) ** 2}
    return {"rel": 5e-7 if case["flavour"] == "mixed" else 6e-15}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
C1 = (3 / 4, -3 / 20, 1 / 60)
C2 = (-49 / 18, 3 / 2, -3 / 20, 1 / 90)
CX = (270 / 720, -27 / 720, 2 / 720)
ALPHA = (0.0, -5 / 9, -153 / 128)
BETA = (1 / 3, 15 / 16, 8 / 15)


def _cut(p, z, y, x):
    """The interior of a padded field, shifted."""
    mz, my, mx = p.shape
    return p[NG + z:mz - NG + z, NG + y:my - NG + y, NG + x:mx - NG + x]


def _unit(axis, k):
    """(z, y, x) shift of k along axis 0 x, 1 y, 2 z."""
    s = [0, 0, 0]
    s[2 - axis] = k
    return s


def _d1(p, axis, inv):
    out = 0
    for k in (1, 2, 3):
        d = _cut(p, *_unit(axis, k)) - _cut(p, *_unit(axis, -k))
        out = d.mul_(C1[k - 1] * inv[axis]) if k == 1 else out.add_(d, alpha=C1[k - 1] * inv[axis])
    return out


def _d2(p, axis, inv):
    s = inv[axis] ** 2
    out = _cut(p, 0, 0, 0) * (C2[0] * s)
    for k in (1, 2, 3):
        out.add_(_cut(p, *_unit(axis, k)), alpha=C2[k] * s)
        out.add_(_cut(p, *_unit(axis, -k)), alpha=C2[k] * s)
    return out


def _dx(p, a, b, inv):
    """Diagonal cross derivative along axes a and b."""
    out = torch.zeros_like(_cut(p, 0, 0, 0))
    for k in (1, 2, 3):
        c = CX[k - 1] * inv[a] * inv[b]
        for sa, sb in ((1, 1), (-1, -1), (1, -1), (-1, 1)):
            sh = [u + v for u, v in zip(_unit(a, sa * k), _unit(b, sb * k))]
            out.add_(_cut(p, *sh), alpha=c * sa * sb)
    return out


def _rhs(p, inv, nu, eta, gamma):
    """Right-hand sides of the eight fields from the padded fields."""
    c = [_cut(f, 0, 0, 0) for f in p]
    u = c[UX:UX + 3]
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    glr = [_d1(p[LNRHO], a, inv) for a in range(3)]
    gs = [_d1(p[SS], a, inv) for a in range(3)]
    gu = [[_d1(p[UX + i], a, inv) for a in range(3)] for i in range(3)]
    div = gu[0][0] + gu[1][1] + gu[2][2]
    out = [None] * 8
    out[LNRHO] = -dot(u, glr) - div

    def second(base):
        """Laplacian and gradient of the divergence of a vector."""
        pure = [[_d2(p[base + i], a, inv) for a in range(3)] for i in range(3)]
        lap = [pure[i][0] + pure[i][1] + pure[i][2] for i in range(3)]
        gd = [pure[i][i] for i in range(3)]
        for i in range(3):
            for k in range(3):
                if i != k:
                    gd[i] = gd[i] + _dx(p[base + k], min(i, k), max(i, k), inv)
        return lap, gd

    ga = [[_d1(p[AX + i], a, inv) if i != a else None for a in range(3)] for i in range(3)]
    b = [ga[2][1] - ga[1][2], ga[0][2] - ga[2][0], ga[1][0] - ga[0][1]]
    del ga
    lap, gd = second(AX)
    j = [(gd[i] - lap[i]) / MU0 for i in range(3)]
    cross = lambda v, w, i: v[(i + 1) % 3] * w[(i + 2) % 3] - v[(i + 2) % 3] * w[(i + 1) % 3]  # noqa: E731
    for i in range(3):
        out[AX + i] = cross(u, b, i) + eta * lap[i]
    e = gamma * c[SS] + (gamma - 1) * (c[LNRHO] - LNRHO0)  # cp = 1
    cs2 = torch.exp(e)  # cs2_sound = 1
    rho = torch.exp(c[LNRHO])
    lap, gd = second(UX)
    s = [[(gu[i][k] + gu[k][i]) / 2 - (div / 3 if i == k else 0) for k in range(3)]
         for i in range(3)]
    for i in range(3):
        out[UX + i] = (-dot(u, gu[i]) - cs2 * (gs[i] + glr[i]) + cross(j, b, i) / rho +
                       nu * (lap[i] + gd[i] / 3 + 2 * dot(s[i], glr)) + ZETA * gd[i])
    heat = eta * MU0 * dot(j, j) + ZETA * rho * div * div
    heat = heat + 2 * rho * nu * sum(dot(s[i], s[i]) for i in range(3))
    del lap, gd, gu, b, j, s
    first = (gamma * sum(_d2(p[SS], a, inv) for a in range(3)) +
             (gamma - 1) * sum(_d2(p[LNRHO], a, inv) for a in range(3)))
    sec = [gamma * gs[i] + (gamma - 1) * glr[i] for i in range(3)]
    thi = [gamma * (gs[i] + glr[i]) - glr[i] for i in range(3)]
    out[SS] = (-dot(u, gs) + heat / (rho * math.exp(LNT0) * cs2) +
               0.001 / rho * (first + dot(sec, thi)))
    return out


def _exact_steps(case, n, fields, nu, eta, forcings=None, after=None):
    """The fields (padded) after the case's steps."""
    as_real = lambda v: float(_real(case["flavour"])[1](v))  # noqa: E731
    ds = [as_real(d) for d in _spacings(n)]
    inv = [as_real(1.0 / d) for d in ds]
    nu, eta, gamma = as_real(nu), as_real(eta), as_real(PHYS["gamma"])
    wall = case.get("wall", 0)
    cur = [f.to(_real(case["flavour"])[0]).double() for f in fields]  # as loaded
    prev = None
    for step in range(case["steps"]):
        dt = as_real(DT)
        if case["kind"] == "cfl":
            umax = float((cur[UX] ** 2 + cur[UY] ** 2 + cur[UZ] ** 2).max()) ** 0.5
            dmin = as_real(min(_spacings(n)))
            dt = min(as_real(CDT) * dmin / (umax + 1.0),
                     as_real(CDTV) * dmin ** 2 / max(nu, eta, gamma))
        for s in range(3):
            rhs = _rhs([_pad(f, wall) for f in cur], inv, nu, eta, gamma)
            for w in range(8):
                r = rhs[w].mul_(BETA[s] * dt).add_(cur[w])
                if s:
                    r.add_(cur[w] - prev[w], alpha=BETA[s] * ALPHA[s] / BETA[s - 1])
            prev, cur = cur, rhs
        if forcings:
            f = forcings[step]
            scale = math.sqrt(dt) * f["magnitude"] * math.sqrt(f["kaver"])  # cs = 1
            x = [torch.arange(m, dtype=torch.float64, device="cuda") * (2.0 * math.pi / m)
                 for m in n]
            ph = (f["k"][2] * x[2][:, None, None] + f["k"][1] * x[1][:, None] +
                  f["k"][0] * x[0] + f["phase"])
            re, im = torch.cos(ph), torch.sin(ph)
            for c in range(3):
                cur[UX + c].add_(scale * (f["re"][c] * re - f["im"][c] * im))
        if after:
            after(cur)
    return [_pad(f, wall) for f in cur]


def exact(case, seed):
    if case["kind"] == "ensemble":
        groups = {}
        for i, m in enumerate(_members(case, seed)):
            out = _exact_steps(case, m["n"], _fields(m["n"], seed, i), m["nu"], m["eta"])
            groups.setdefault(m["n"][0], []).append(torch.stack([_cut(f, 0, 0, 0) for f in out]))
        return [torch.stack(g) for g in groups.values()]
    n = _n(case)
    values = []

    def after(cur):
        u = torch.sqrt(cur[UX] ** 2 + cur[UY] ** 2 + cur[UZ] ** 2)
        of_u = [float(u.max()), float(u.min()), float((u * u).sum())]
        rms_exp = float(torch.exp(2 * cur[LNRHO]).sum())
        if case["kind"] == "forced":
            values.append(of_u + [rms_exp])
        elif case["kind"] == "snapshot":
            values.append(of_u[:1])
        else:
            for f in cur:
                of_u += [float(f.max()), float(f.min()), float((f * f).sum())]
            values.append(of_u + [rms_exp])

    forcings = _forcings(case, seed) if case["kind"] == "forced" else None
    wanted = case["kind"] in ("forced", "snapshot", "diagnostics")
    fields = _exact_steps(case, n, _fields(n, seed), PHYS["nu_visc"], PHYS["eta"], forcings,
                          after if wanted else None)
    if wanted:
        return dict(fields=fields, values=np.array(values, dtype=np.float64))
    return dict(fields=fields)
