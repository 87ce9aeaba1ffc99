"""Reductions on rows of every remainder, and on values that no comparison holds."""
import math

import numpy as np
import pytest

from astaroth_b200 import Device, abi

pytestmark = pytest.mark.gpu
U = (abi.VTXBUF_UUX, abi.VTXBUF_UUY, abi.VTXBUF_UUZ)


# a lane takes four vertices of a row at a time: rows shorter than a warp, of whole
# groups of four, and of each remainder
@pytest.mark.parametrize("nx", [3, 31, 33, 96, 127, 128, 130, 257])
@pytest.mark.parametrize("flavour", ["sp", "dp", "mixed"])
def test_rows_of_every_remainder(flavour, nx):
    """Every kind of one field and of a vector against numpy in FP64: MAX and MIN
    exactly, sums to 1e-12 (FP64 sums of under 3000 terms in another order err by
    at most 3000 * 1.1e-16 of the sum of magnitudes); the passes over several
    fields return what passes of their own return, bit for bit."""
    prec = abi.PRECISIONS[flavour]
    info = abi.make_info(prec, nx, 3, 4)
    rng = np.random.default_rng(nx)
    shape = (10, 9, nx + 6)
    fields = [rng.standard_normal(shape).astype(prec.np_dtype) for _ in range(8)]
    g = abi.NGHOST
    f = [x[g:-g, g:-g, g:-g].astype(np.float64) for x in fields]
    length = np.sqrt(f[1] ** 2 + f[2] ** 2 + f[3] ** 2)
    kinds = (abi.RTYPE_MAX, abi.RTYPE_MIN, abi.RTYPE_RMS)

    def check(got, want, kind):
        if kind in kinds[:2]:
            assert abs(got - want) <= 4e-16 * abs(want), (got, want)
        else:
            assert abs(got - want) <= 1e-12 * abs(want), (got, want)

    def wanted(x, kind):
        return {abi.RTYPE_MAX: x.max(), abi.RTYPE_MIN: x.min()}.get(kind, (x * x).sum())

    with Device(flavour, info) as dev:
        dev.load_mesh(abi.HostMesh(prec, info, fields))
        alone = [dev.reduce_vec_double(k, *U) for k in kinds]  # a pass of its own
        for k, got in zip(kinds, alone):
            check(got, wanted(length, k), k)
        for w in range(8):  # from the second on, passes over all they read
            for k in kinds:
                check(dev.reduce_scal_double(k, w), wanted(f[w], k), k)
        dev.load_mesh(abi.HostMesh(prec, info, fields))
        assert [dev.reduce_vec_double(k, *U) for k in kinds] == alone
        check(dev.reduce_scal_double(abi.RTYPE_RMS_EXP, 0), np.exp(2 * f[0]).sum(), None)
        check(dev.reduce_vec_double(abi.RTYPE_SUM, *U), length.sum(), None)


@pytest.mark.parametrize("flavour", ["sp", "dp", "mixed"])
def test_nan_and_infinite_lengths(flavour):
    """NaN values take no part in MAX and MIN (all NaN: the identities remain),
    infinite ones do, as each length compared on its own would give."""
    prec = abi.PRECISIONS[flavour]
    n = 5
    info = abi.make_info(prec, n, n, n)
    fields = [np.full((n + 6,) * 3, np.nan, prec.np_dtype) for _ in range(8)]
    with Device(flavour, info) as dev:
        dev.load_mesh(abi.HostMesh(prec, info, fields))
        assert dev.reduce_vec_double(abi.RTYPE_MAX, *U) == -math.inf
        assert dev.reduce_vec_double(abi.RTYPE_MIN, *U) == math.inf
        assert math.isnan(dev.reduce_vec_double(abi.RTYPE_RMS, *U))
        for w in (1, 2, 3):
            fields[w][5, 5, 5] = 3.0 if w == 1 else 0.0
        dev.load_mesh(abi.HostMesh(prec, info, fields))
        assert dev.reduce_vec_double(abi.RTYPE_MAX, *U) == 3.0
        assert dev.reduce_vec_double(abi.RTYPE_MIN, *U) == 3.0
        fields[1][5, 5, 5] = -np.inf
        dev.load_mesh(abi.HostMesh(prec, info, fields))
        assert dev.reduce_vec_double(abi.RTYPE_MAX, *U) == math.inf
        assert dev.reduce_vec_double(abi.RTYPE_MIN, *U) == math.inf
