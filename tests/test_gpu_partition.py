"""The whole-box wall fill at the sizes where it can go wrong."""
import math

import numpy as np
import pytest

from astaroth_b200 import Device, abi, init

pytestmark = pytest.mark.gpu
FLAVOURS = ("sp", "dp", "mixed")


def mesh_info(prec, n, **more):
    return abi.make_info(prec, *n, dsx=2 * math.pi / n[0], dsy=2 * math.pi / n[1],
                         dsz=2 * math.pi / n[2], gamma=5 / 3, nu_visc=5e-3, eta=5e-3, **more)


@pytest.mark.parametrize("n", [(4, 4, 4), (8, 5, 6), (21, 9, 4), (124, 7, 5), (130, 4, 9)])
@pytest.mark.parametrize("bc", [abi.AC_BOUNDCOND_SYMMETRIC, abi.AC_BOUNDCOND_ANTISYMMETRIC])
@pytest.mark.parametrize("flavour", FLAVOURS)
def test_whole_box_walls_equal_field_by_field(flavour, bc, n):
    """The one-launch wall fill (rows of whole sectors, nx % 4 == 0, and others)
    equals the fill of one field at a time, bit for bit, lo parts included."""
    info = mesh_info(abi.PRECISIONS[flavour], n, bc_type_top_x=bc)
    rng = np.random.default_rng(5)
    # doubles: in the mixed build every vertex then has a lo part
    fields = [rng.standard_normal(tuple(m + 6 for m in n[::-1])) for _ in range(8)]
    got = []
    for whole in (True, False):
        with Device(flavour, info) as dev:
            for w, f in enumerate(fields):
                dev.load_double(w, f)
            lo, hi = dev.full_box()
            out = abi.int3(-1, -1, -1)
            if whole:
                rc = dev.lib.acDeviceGeneralBoundconds(dev.handle, 0, lo, hi, info, out)
                assert rc == abi.AC_SUCCESS
            else:
                for w in range(8):
                    rc = dev.lib.acDeviceGeneralBoundcondStep(dev.handle, 0, w, lo, hi, info, out)
                    assert rc == abi.AC_SUCCESS
            got.append([dev.store_double(w) for w in range(8)])
    for w in range(8):
        assert np.array_equal(got[0][w], got[1][w]), w
