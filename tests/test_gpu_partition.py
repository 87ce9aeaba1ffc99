"""The split of a launch's tile columns over the CTAs, the ghost images that a
substep writes, the whole-box wall fill and the direct copies of a mesh that lies
in GPU memory, at the sizes where each can go wrong."""
import ctypes as C
import math

import numpy as np
import pytest

from astaroth_b200 import Device, abi, init

pytestmark = pytest.mark.gpu
FLAVOURS = ("sp", "dp", "mixed")


def mesh_info(prec, n, **more):
    return abi.make_info(prec, *n, dsx=2 * math.pi / n[0], dsy=2 * math.pi / n[1],
                         dsz=2 * math.pi / n[2], gamma=5 / 3, nu_visc=5e-3, eta=5e-3, **more)


# the smallest mesh; slabs of few planes; slabs and shares of what they leave, some
# across two columns and more; z segments; whole columns, alone and with a partial
# wave after them. Each library takes each of these forms at one of the sizes on a
# GPU of 148 SMs: test_host_side.py (test_the_split_takes_every_form).
SPLIT_SIZES = [(3, 3, 3), (32, 30, 40), (97, 50, 75), (200, 190, 33), (420, 160, 9),
               (200, 168, 48), (200, 108, 48), (64, 228, 52), (128, 444, 7)]


@pytest.mark.parametrize("n", SPLIT_SIZES)
@pytest.mark.parametrize("flavour", FLAVOURS)
def test_every_plane_of_every_column_once(flavour, n):
    """A step through each tile configuration (each splits the mesh differently)
    equals the step taken as sub-boxes of two planes, bit for bit."""
    prec = abi.PRECISIONS[flavour]
    info = mesh_info(prec, n)
    fields = init.workload_fields(*n, prec.np_dtype, seed=3, amplitude=1e-2, velocity_mode=0.1)
    host = abi.HostMesh(prec, info, fields)
    g, dt = abi.NGHOST, 1e-3

    def stepped(dev, boxes):
        dev.load_mesh(host)
        for s in range(3):
            dev.periodic_boundconds()
            for lo, hi in boxes:
                dev.integrate_substep(s, dt, lo, hi)
            dev.swap_buffers()
        out = abi.HostMesh(prec, info)
        dev.store_mesh(out)
        assert dev.status() == 0
        return [out.interior(w).copy() for w in range(8)]

    with Device(flavour, info) as dev:
        slabs = [(abi.int3(g, g, g + z), abi.int3(g + n[0], g + n[1], g + min(z + 2, n[2])))
                 for z in range(0, n[2], 2)]
        want = stepped(dev, slabs)
        for cfg in range(dev.solve_config()[1]):
            dev.set_solve_config(cfg)
            got = stepped(dev, [dev.interior_box()])
            for w in range(8):
                assert np.array_equal(got[w], want[w]), (cfg, w)


# the smallest mesh that writes images (6 an axis), meshes below it, rows and
# columns that end within a tile, every vertex near two faces, a long axis
@pytest.mark.parametrize("n", [(6, 6, 6), (5, 9, 12), (7, 6, 11), (33, 13, 8), (40, 12, 50),
                               (64, 64, 64), (200, 9, 7)])
@pytest.mark.parametrize("flavour", FLAVOURS)
def test_whole_steps_equal_the_substep_loop(flavour, n):
    """Whole steps, whose substeps write the ghost images on small meshes, leave
    the very state, ghosts and lo parts included, that ghost fills, substeps and
    buffer swaps leave."""
    prec = abi.PRECISIONS[flavour]
    info = mesh_info(prec, n)
    fields = init.workload_fields(*n, prec.np_dtype, seed=4, amplitude=1e-2, velocity_mode=0.1)
    host, dt = abi.HostMesh(prec, info, fields), 1e-3

    def loop(dev):
        for _ in range(3):
            for s in range(3):
                dev.periodic_boundconds()
                dev.integrate_substep(s, dt)
                dev.swap_buffers()

    def steps(dev):
        for _ in range(3):
            dev.integrate_step(dt)

    got = []
    for advance in (loop, steps, lambda dev: dev.integrate_steps(dt, 3)):
        with Device(flavour, info) as dev:
            dev.load_mesh(host)
            advance(dev)
            got.append([dev.store_double(w) for w in range(8)])
            dev.periodic_boundconds()
            got[-1] += [dev.store_double(w) for w in range(8)]
            assert dev.status() == 0
    for other in got[1:]:
        for w in range(16):
            assert np.array_equal(got[0][w], other[w]), w


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


@pytest.mark.parametrize("n,start,count", [((5, 4, 3), 0, None), ((37, 29, 23), 1234, 5 * 43 + 17),
                                           ((64, 12, 7), 0, None)])
@pytest.mark.parametrize("flavour", FLAVOURS)
def test_mesh_in_gpu_memory_copies_like_a_host_mesh(flavour, n, start, count):
    """Load and store of a whole mesh, or of a flat range that starts and ends
    within a row, from and to arrays in GPU memory."""
    import torch

    prec = abi.PRECISIONS[flavour]
    info = mesh_info(prec, n)
    shape = tuple(m + 6 for m in n[::-1])
    total = math.prod(shape)
    count = total if count is None else count
    rng = np.random.default_rng(7)
    fields = [rng.standard_normal(shape).astype(prec.np_dtype) for _ in range(8)]
    on_gpu = [torch.from_numpy(f).cuda() for f in fields]
    back = [torch.full_like(t, 7.0) for t in on_gpu]

    def mesh(tensors):
        m = abi.mesh_type(prec)()
        m.info = info
        for w, t in enumerate(tensors):
            m.vertex_buffer[w] = C.cast(C.c_void_p(t.data_ptr()), C.POINTER(prec.real))
        return m

    mx, my = shape[2], shape[1]
    at = abi.int3(start % mx, start // mx % my, start // (mx * my))
    torch.cuda.synchronize()
    with Device(flavour, info) as dev:
        lib = dev.lib
        assert lib.acDeviceLoadMeshWithOffset(dev.handle, 0, mesh(on_gpu), at, at, count) == 0
        dst = mesh(back)
        assert lib.acDeviceStoreMeshWithOffset(dev.handle, 0, at, at, count, C.byref(dst)) == 0
        dev.synchronize()
        host = abi.HostMesh(prec, info)
        dev.store_mesh(host)
        # one field on its own
        alone = [torch.full_like(t, 7.0) for t in on_gpu]
        torch.cuda.synchronize()
        dst = mesh(alone)
        assert lib.acDeviceStoreVertexBufferWithOffset(dev.handle, 0, 5, at, at, count,
                                                       C.byref(dst)) == 0
        dev.synchronize()
    for w in range(8):
        want = np.full(total, 7.0, prec.np_dtype)
        want[start:start + count] = fields[w].reshape(-1)[start:start + count]
        assert np.array_equal(back[w].cpu().numpy().reshape(-1), want), w
        want = np.zeros(total, prec.np_dtype)
        want[start:start + count] = fields[w].reshape(-1)[start:start + count]
        assert np.array_equal(host.fields[w].reshape(-1), want), w
    assert np.array_equal(alone[5].cpu().numpy(), back[5].cpu().numpy())
    assert all(bool((alone[w] == 7.0).all()) for w in range(8) if w != 5)
