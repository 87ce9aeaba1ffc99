"""The mixed build's right-hand sides at their own rounding: terms whose operations
could be ordered or scaled so that their errors add up from step to step."""
import math

import numpy as np
import pytest

from astaroth_b200 import Device, abi, init

pytestmark = pytest.mark.gpu
N, G = 64, abi.NGHOST


def f32(x):
    return np.asarray(x, np.float64).astype(np.float32).astype(np.float64)


def rate(fields, w, inv, **params):
    """d/dt of field w of a periodic N^3 mesh of float fields, from one substep whose
    beta dt is 1/4, exactly; inv: 1 / ds of every axis."""
    info = abi.make_info(abi.MIXED, N, dsx=1.0 / inv, dsy=1.0 / inv, dsz=1.0 / inv, **params)
    for axis in "xyz":
        abi.set_real(info, f"inv_ds{axis}", inv)
    with Device("mixed", info) as dev:
        dev.load_mesh(abi.HostMesh(abi.MIXED, info, [f.astype(np.float32) for f in fields]))
        dev.periodic_boundconds()
        before = dev.store_double(w)
        dev.integrate_substep(0, 0.75)
        dev.swap_buffers()
        after = dev.store_double(w)
        assert dev.status() == 0
    return 4.0 * (after - before)[G:-G, G:-G, G:-G]


def shifted(f, axis, k):
    """Interior of a padded field [z, y, x], shifted by k along axis 0 x, 1 y, 2 z."""
    s = [0, 0, 0]
    s[2 - axis] = k
    return f[tuple(slice(G + d, G + N + d) for d in s)]


def first(f, axis, inv, rnd):
    d = [rnd(shifted(f, axis, k) - shifted(f, axis, -k)) for k in (1, 2, 3)]
    if rnd is f32:
        s1, r2 = float(f32(0.75 * inv)), float(f32(-1 / 5))
        r3 = float(f32((inv / s1 - 2 - 4 * r2) / 6))
        return f32(s1 * f32(f32(d[0] + r2 * d[1]) + r3 * d[2]))
    return inv * (0.75 * d[0] - 0.15 * d[1] + d[2] / 60)


def test_continuity_rounds_the_divergence_once():
    """d lnrho/dt = -(u . grad lnrho + div u): no noisier than in this order of
    operations with each result rounded to a float. (Adding the products to the
    divergence one by one is 12 % noisier: 1.71e-9 instead of 1.52e-9 at 128^3.)"""
    inv = float(np.float32(N / (2 * math.pi)))
    fields = init.workload_fields(N, N, N, np.float32, seed=1, amplitude=1e-3, velocity_mode=0.1)
    f = [np.asarray(x, np.float64) for x in fields]

    def continuity(rnd):
        u = [shifted(f[1 + i], 0, 0) for i in range(3)]
        gl = [first(f[0], i, inv, rnd) for i in range(3)]
        gu = [first(f[1 + i], i, inv, rnd) for i in range(3)]
        div = rnd(rnd(gu[0] + gu[1]) + gu[2])
        products = rnd(u[0] * gl[0] + rnd(u[1] * gl[1] + rnd(u[2] * gl[2])))
        return -rnd(products + div)

    exact = continuity(lambda x: x)
    rms = lambda e: float(np.sqrt(np.mean(e * e)))  # noqa: E731
    got, want = rms(rate(fields, abi.VTXBUF_LNRHO, inv) - exact), rms(continuity(f32) - exact)
    print(f"continuity: rms error {got:.3e}, in this order {want:.3e}")
    # 2.6e5 vertices: the rms of either is known to 0.3 %
    assert got <= 1.02 * want


def test_first_derivatives_have_no_factor():
    """With lnrho = 0 its rate is -div u. Of a smooth u it is off by one factor where
    the rounded coefficients do not add up to 1 / ds (-3.8e-8 here with 3/4 / ds, -1/5
    and 1/45 rounded one by one). The last coefficient makes up for the others to half
    a unit in its own last place."""
    inv = float(np.float32(N / (2 * math.pi)))
    x = np.arange(-G, N + G) * (2 * math.pi / N)
    z, y, x = np.meshgrid(x, x, x, indexing="ij")
    fields = [np.zeros_like(x) for _ in range(8)]
    for i, k in enumerate(((1, 2, -1), (2, 1, 1), (-1, 1, 2))):
        fields[abi.VTXBUF_UUX + i] = f32(0.1 * np.sin(k[0] * x + k[1] * y + k[2] * z + i))
    got = rate(fields, abi.VTXBUF_LNRHO, inv)
    want = -sum(first(fields[abi.VTXBUF_UUX + i], i, inv, lambda v: v) for i in range(3))
    factor = float(((got - want) * want).sum() / (want * want).sum())
    # d3 is 6 h f' of the sum's 4/3 h f'; its coefficient's ulp is 2^-29. Between d1 and
    # d3 the share of d3 falls with the wavenumber, as 1 - 4/3 (k h)^2. The roundings of
    # the operations, 2e-8 each, leave 1e-10 of the mean over 2.6e5 vertices
    bound = 6 * 2.0 ** -30 / (4 / 3) + 3.8e-8 * 4 / 3 * (2 * 2 * math.pi / N) ** 2 + 1e-10
    print(f"first derivatives: off by {factor:.2e}, bound {bound:.2e}")
    assert abs(factor) <= bound


def test_ohmic_heating_has_no_factor():
    """With u = lnrho = s = 0 the entropy's rate is eta mu0 j^2 / (rho T), j of second
    derivatives. It is off by one factor where their scale 3/2 / ds^2 is rounded, at
    a spacing where that rounding is nearly as large as it gets. What remains
    is the rounding of one product of parameters and that of the stencil's
    coefficients: -1/10 and 1/135 as floats leave a smooth derivative off by 1.1e-8."""
    inv = np.float32(13.0)
    off = lambda v: float(np.float32(1.5 * float(v) ** 2)) / (1.5 * float(v) ** 2) - 1  # noqa: E731
    while abs(off(inv)) < 5.5e-8:
        inv = np.nextafter(inv, np.float32(14.0))
    inv = float(inv)
    rng = np.random.default_rng(3)
    fields = [np.zeros((N + 2 * G,) * 3) for _ in range(8)]
    for w in (abi.VTXBUF_AX, abi.VTXBUF_AY, abi.VTXBUF_AZ):
        a = rng.uniform(-1e-3, 1e-3, (N,) * 3).astype(np.float32).astype(np.float64)
        fields[w] = np.pad(a, G, mode="wrap")
    eta, mu0 = 2.0 ** -8, 1.0
    got = rate(fields, abi.VTXBUF_ENTROPY, inv, eta=eta, mu0=mu0, lnT0=0.0, lnrho0=0.0,
               gamma=5 / 3, nu_visc=5e-3, cs_sound=1.0, cp_sound=1.0)
    A = fields[abi.VTXBUF_AX:abi.VTXBUF_AZ + 1]
    pure = [[sum(c * (shifted(A[i], a, k) + shifted(A[i], a, -k) - 2 * shifted(A[i], a, 0))
                 for k, c in ((1, 1.5), (2, -0.15), (3, 1 / 90))) for a in range(3)]
            for i in range(3)]

    def cross(f, a, b):
        out = 0
        for k, c in ((1, 270 / 720), (2, -27 / 720), (3, 2 / 720)):
            for sa, sb in ((1, 1), (-1, -1), (1, -1), (-1, 1)):
                s = [0, 0, 0]
                s[2 - a], s[2 - b] = sa * k, sb * k
                out = out + c * sa * sb * f[tuple(slice(G + d, G + N + d) for d in s)]
        return out

    j2 = 0
    for i in range(3):
        j = sum(cross(A[k], min(i, k), max(i, k)) for k in range(3) if k != i)
        j2 = j2 + (j - sum(pure[i][a] for a in range(3) if a != i)) ** 2
    want = eta * mu0 * j2 * (inv * inv / mu0) ** 2
    factor = float(((got - want) * want).sum() / (want * want).sum())
    unit = 2.0 * math.frexp(1.5 * inv * inv)[0]
    k = eta / mu0 * unit * unit
    bound = abs(float(np.float32(k)) / k - 1) + 2 * 1.1e-8
    print(f"heating: off by {factor:.2e}, bound {bound:.2e}, the scale alone {2 * off(inv):.2e}")
    assert bound < 0.5 * abs(2 * off(inv))
    assert abs(factor) <= bound
