"""The library's host code (an ensemble's schedule, uploads, graphs and tuner; the
route of a mesh transfer) on a stand-in CUDA runtime (fake_cudart.c): no GPU, no
kernel runs."""
import os
import subprocess
import sys
import textwrap

import pytest

from astaroth_b200 import abi
from test_gpu_partition import SPLIT_SIZES

TESTS = os.path.dirname(os.path.abspath(__file__))
FLAVOURS = ("sp", "dp", "mixed")

PREAMBLE = """
import ctypes, sys
from astaroth_b200 import Ensemble, abi
from astaroth_b200.device import AcError
fake = ctypes.CDLL(None)
flavour, cache = sys.argv[1], sys.argv[2]
prec = abi.PRECISIONS[flavour]
def ensemble(n=(40, 24, 32)):
    return Ensemble(flavour, [abi.make_info(prec, n[0] + 8 * k, n[1], n[2]) for k in range(3)])
"""


@pytest.fixture(scope="module")
def fake_runtime(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    lib = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", f"-I{cuda}/include",
                    os.path.join(TESTS, "fake_cudart.c"), "-o", lib], check=True)
    return lib


def run(fake_runtime, tmp_path, flavour, body):
    env = dict(os.environ, LD_PRELOAD=fake_runtime, PYTHONPATH=abi.REPO)
    r = subprocess.run([sys.executable, "-c", PREAMBLE + textwrap.dedent(body), flavour,
                        str(tmp_path / "tune.txt")], env=env, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_tables_are_in_place_before_a_launch(fake_runtime, tmp_path, flavour):
    """Nothing is launched on the ensemble's non-blocking stream while an upload
    or a memset of another stream may still be pending."""
    run(fake_runtime, tmp_path, flavour, """
        e = ensemble()
        e.integrate_step(1e-3)
        e.set_schedule(1, 16)
        e.integrate_step(1e-3)
        e.auto_optimize(cache)
        assert fake.fake_launches() > 12
        assert fake.fake_unordered_launches() == 0
    """)


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_a_refused_schedule_leaves_the_one_in_use(fake_runtime, tmp_path, flavour):
    """A schedule whose tables cannot be allocated is refused; the ensemble keeps
    its tables, its schedule and its graphs, and goes on."""
    run(fake_runtime, tmp_path, flavour, """
        e = ensemble()
        e.set_schedule(1, 16)
        e.integrate_steps(1e-3, 2)
        live, graphs = fake.fake_live_allocations(), fake.fake_graphs_instantiated()
        fake.fake_fail_malloc(0)
        try:
            e.set_schedule(2, 8)
            sys.exit("accepted")
        except AcError:
            pass
        assert fake.fake_live_allocations() == live
        assert e.schedule() == (1, 16)
        e.integrate_steps(1e-3, 2)
        assert fake.fake_graphs_instantiated() == graphs
        e.set_schedule(2, 8)
        assert e.schedule() == (2, 8) and fake.fake_live_allocations() == live
        e.destroy()
        assert fake.fake_live_allocations() == 0
    """)


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_a_graph_is_replayed_for_its_own_time_step_only(fake_runtime, tmp_path, flavour):
    """A captured step holds its time step: the next value of the library's
    precision takes a graph of its own (one for each buffer parity)."""
    run(fake_runtime, tmp_path, flavour, """
        import numpy as np
        e, dt = ensemble(), prec.np_dtype(1e-3)
        e.integrate_steps(dt, 6)  # both parities
        graphs = fake.fake_graphs_instantiated()
        e.integrate_steps(dt, 4)
        assert fake.fake_graphs_instantiated() == graphs
        e.integrate_steps(np.nextafter(dt, prec.np_dtype(1)), 2)
        assert fake.fake_graphs_instantiated() == graphs + 2
    """)


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_a_new_ensemble_reports_the_schedule_it_runs(fake_runtime, tmp_path, flavour):
    """Whole columns of the first configuration."""
    run(fake_runtime, tmp_path, flavour, """
        assert ensemble().schedule() == (0, 0)
    """)


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_a_choice_timed_on_other_kernels_is_not_taken(fake_runtime, tmp_path, flavour):
    """The tuner's cache: an entry that names only the precision and the sizes, as
    older ones do, misses; the entry of this library hits."""
    run(fake_runtime, tmp_path, flavour, """
        old = flavour + "|1*40x24x32|1*48x24x32|1*56x24x32 1 64\\n"
        open(cache, "w").write(old)
        e = ensemble()
        e.auto_optimize(cache)
        assert e.schedule() == (2, 16)  # the last one timed (see cudaEventElapsedTime)
        text = open(cache).read()
        assert text.startswith(old) and len(text.split()) == 6
        launches = fake.fake_launches()
        other = ensemble()
        other.auto_optimize(cache)
        assert other.schedule() == (2, 16) and fake.fake_launches() == launches
    """)


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_a_mesh_that_is_not_all_mapped_is_refused(fake_runtime, tmp_path, flavour):
    """A mesh in address space that the program maps itself is copied, not read and
    written in place by a kernel: the driver reports the whole reservation as the
    pointer's range, and only a copy refuses what is not mapped of it."""
    run(fake_runtime, tmp_path, flavour, """
        from astaroth_b200 import Device
        n = (40, 24, 32)
        info = abi.make_info(prec, *n)
        cells = (n[0] + 6) * (n[1] + 6) * (n[2] + 6)
        field = cells * ctypes.sizeof(prec.real)
        host = (ctypes.c_char * (9 * field))()
        base = ctypes.addressof(host)

        def mesh(at):
            m = abi.mesh_type(prec)()
            m.info = info
            for w in range(8):
                m.vertex_buffer[w] = ctypes.cast(at + w * field, ctypes.POINTER(prec.real))
            return m

        def load_and_store(dev, m):
            before = fake.fake_launches()
            rc = (dev.lib.acDeviceLoadMesh(dev.handle, 0, m),
                  dev.lib.acDeviceStoreMesh(dev.handle, 0, ctypes.byref(m)))
            return rc, fake.fake_launches() - before

        dev = Device(flavour, info)
        plain = ctypes.c_void_p()
        fake.cudaMalloc(ctypes.byref(plain), ctypes.c_size_t(8 * field))
        assert load_and_store(dev, mesh(plain.value)) == ((0, 0), 2)
        # all of it mapped: a copy and a kernel for each field
        fake.fake_reserve(ctypes.c_void_p(base), ctypes.c_size_t(9 * field), ctypes.c_size_t(8 * field))
        assert load_and_store(dev, mesh(base)) == ((0, 0), 16)
        # the last field not
        fake.fake_reserve(ctypes.c_void_p(base), ctypes.c_size_t(9 * field), ctypes.c_size_t(8 * field - 4))
        rc, launches = load_and_store(dev, mesh(base))
        assert rc == (1, 1) and launches > 2
    """)


@pytest.mark.parametrize("flavour", FLAVOURS)
def test_the_split_takes_every_form(fake_runtime, tmp_path, flavour):
    """The sizes at which test_gpu_partition.py compares the split of the columns
    reach, between them and the tile configurations, every form that it can take."""
    run(fake_runtime, tmp_path, flavour, f"sizes = {SPLIT_SIZES}\n" + """
from astaroth_b200 import Device
forms = set()
for n in sizes:
    dev = Device(flavour, abi.make_info(prec, *n))
    for cfg in range(dev.solve_config()[1]):
        dev.set_solve_config(cfg)
        dev.integrate_substep(0, 1e-3)
        w = (ctypes.c_int * 30)()
        fake.fake_last_solve(w)
        assert tuple(w[3:6]) == n and w[21] == n[2]  # Layout::nx, ny, nz; SolveGeom::nzr
        nfull, rem0, rem, slabs, slab_planes, left, zseg, seg_tasks = w[22:30]
        if seg_tasks:
            forms.add("segments")
            continue
        if nfull:
            forms.add("whole, then slabs" if rem else "whole")
        elif slabs > 1:
            forms.add("slabs")
        if left:
            forms.add("shares")
            if rem > 148 - slabs * rem:
                forms.add("shares across columns")
    dev.destroy()
want = {"segments", "whole, then slabs", "whole", "slabs", "shares", "shares across columns"}
assert forms == want, want - forms
""")
