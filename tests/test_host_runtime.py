"""The engine's host code over a CUDA runtime without a device
(fake_cudart.cpp: memory is the host's, launches are checked and written down,
no kernel runs): what one GPU cannot show (several devices) and what a GPU
should not be made to show (launches that are refused)."""
import ctypes
import glob
import os
import subprocess

import pytest

import helpers
from dnlPython import _abi, meshes
from dnlPython.engine import Engine

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    objs = glob.glob(os.path.join(helpers.PKG, "lib", "obj", "*.o"))
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not objs or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime_api.h")):
        pytest.skip("the build's object files or the CUDA headers are not here")
    out = str(tmp_path_factory.mktemp("fake") / "libdnlgpu_fake.so")
    # -Bsymbolic: the engine's calls reach the fake also where a CUDA runtime is loaded
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I",
                    os.path.join(cuda, "include"), "-o", out, os.path.join(HERE, "fake_cudart.cpp")] + objs,
                   check=True)
    return out


@pytest.fixture
def fake(fake_path, monkeypatch):
    monkeypatch.setattr(_abi, "LIB_PATH", fake_path)
    monkeypatch.setattr(_abi, "_lib", None)
    lib = _abi.load_library()
    lib.fake_launch.restype = ctypes.c_char_p
    lib.fake_used.restype = ctypes.c_size_t
    lib.fake_reset(2, ctypes.c_size_t(1 << 40))
    return lib


def launches(lib, kernel):
    """(grid.x, grid.y, threads, dynamic shared memory, device) of the launches of a kernel."""
    out = []
    for i in range(lib.fake_launches()):
        v = (ctypes.c_int * 5)()
        if kernel in lib.fake_launch(i, v).decode():
            out.append(tuple(v))
    return out


@pytest.mark.parametrize("precision,variant", [(_abi.PREC_FP64, v) for v in range(_abi.NUM_VARIANTS)]
                         + [(_abi.PREC_MIXED, v) for v in range(_abi.NUM_VARIANTS)])
def test_engines_on_two_devices_in_one_process(fake, precision, variant):
    """Every element-pass variant launches on the second device as on the
    first: the shared-memory opt-in of a kernel holds per device."""
    d = meshes.hex_block(3, 3, 3, precision=precision)
    for device in (0, 1, 0):
        fake.fake_set_device(device)
        fake.fake_clear_log()
        with Engine(d) as e:
            e.init()
            e.set_variant(variant)
            fake.fake_clear_log()
            e.run(max_incs=2)
            assert [x[4] for x in launches(fake, "k_element")] == [device] * 2


@pytest.mark.parametrize("call", ["dnl_mlp_forward", "dnl_mlp_gradients"])
def test_network_calls_on_two_devices_in_one_process(fake, call):
    net, grad = _abi.Mlp(), _abi.Mlp()
    x = (ctypes.c_float * 5)()
    y = (ctypes.c_float * 1)()
    for device in (0, 1):
        fake.fake_set_device(device)
        if call == "dnl_mlp_forward":
            rc = fake.dnl_mlp_forward(ctypes.byref(net), x, 1, y, None)
        else:
            rc = fake.dnl_mlp_gradients(ctypes.byref(net), x, y, 1, ctypes.byref(grad), y, None)
        assert rc == _abi.DNL_OK, fake.dnl_engine_last_error(None)


def _refused(call):
    with pytest.raises(_abi.EngineError) as x:
        call()
    assert x.value.code == -2 and "launch failed" in str(x.value)


@pytest.mark.parametrize("kernel", ["k_element_once", "k_nodal", "k_courant_finish"])
@pytest.mark.parametrize("timed", [False, True])
def test_a_refused_launch_is_an_error_of_every_run(fake, kernel, timed):
    """A kernel that cannot be launched fails the run that captures it and the
    next one too (no graph without it is kept); launched again, the run goes on."""
    with Engine(meshes.hex_block(3, 3, 3)) as e:
        e.init()
        e.set_variant(0)
        e.set_timing(timed)
        fake.fake_refuse(kernel.encode())
        for _ in range(2):
            fake.fake_clear_log()
            _refused(lambda: e.run(max_incs=20))
            # (kernel by kernel, those before it have been queued)
            assert timed or [k for k in ("k_element", "k_nodal", "k_courant") if launches(fake, k)] == []
        variant = e.variant()[0]
        _refused(lambda: e.autotune(2))
        assert e.variant()[0] == variant
        fake.fake_refuse(b"")
        fake.fake_clear_log()
        e.run(max_incs=20)
        assert len(launches(fake, kernel)) > 0


def test_a_refused_launch_is_an_error_of_the_start_and_of_a_pass(fake):
    with Engine(meshes.hex_block(3, 3, 3)) as e:
        for kernel in (b"k_element_start", b"k_courant", b"k_control", b"k_element_once"):
            fake.fake_refuse(kernel)
            _refused(e.init)
        fake.fake_refuse(b"")
        e.init()
        fake.fake_refuse(b"k_gather")
        _refused(lambda: e.element_pass(1e-9))


def test_energies_of_more_instances_than_a_grid_has_rows(fake):
    """65,535 is where the second and third dimension of a grid end."""
    d = meshes.hex_block(1, 1, 1)
    with Engine([d] * 65_600) as e:
        e.init()
        e.energies(65_599)
        e.set_items([(_abi.ITEM_KINETIC, f, 65_599) for f in (_abi.NODE_SPEED, _abi.NODE_SPEED_PREV)])
        e.gather_items()


def test_energies_launch_and_keep_what_they_need(fake):
    """One instance's energies are that instance's work, tiny instances are a
    block each, and an instance adds no kilobytes of partial sums to a batch."""
    d = meshes.hex_block(1, 1, 1)
    used = {}
    for n in (1000, 2000):
        before = fake.fake_used(0)
        with Engine([d] * n) as e:
            used[n] = fake.fake_used(0) - before
            e.init()
            fake.fake_clear_log()
            e.energies(7)
            assert [x[0] for x in launches(fake, "k_energy")] == [1, 1]
            e.set_items([(_abi.ITEM_KINETIC, _abi.NODE_SPEED, k) for k in (0, n - 1)])
            fake.fake_clear_log()
            e.gather_items()
            assert [x[0] for x in launches(fake, "k_energy")] == [n, n]
    # 8 points and nodes, the control block and the tables: about 6 KB
    assert (used[2000] - used[1000]) / 1000 < 8192
    # an ordinary model: a block per 256 points, at most 256
    with Engine([meshes.hex_block(9, 10, 11), d]) as e:
        e.init()
        fake.fake_clear_log()
        e.energies(1)
        assert launches(fake, "k_energy_parts")[0][0] == (8 * 990 + 255) // 256
    with Engine(meshes.hex_block(25, 25, 25)) as e:
        e.init()
        fake.fake_clear_log()
        e.energies()
        assert launches(fake, "k_energy_parts")[0][0] == 256


@pytest.mark.parametrize("mesh,element", [(lambda: meshes.hex_block(3, 3, 3), "k_element_stage"),
                                          (lambda: meshes.quad_block(5, 5), "k_element")], ids=["hex", "quad"])
def test_autotune_after_set_variant_chooses_again(fake, mesh, element):
    """A variant asked for holds until the autotuner is asked: then a small
    model runs its increments in cooperative launches again."""
    with Engine(mesh()) as e:
        e.init()
        for asked in (False, True, False):
            if asked:
                e.set_variant(6)
            else:
                e.autotune(2)
            for _ in range(2):
                fake.fake_clear_log()
                e.run(max_incs=3)
                assert [bool(launches(fake, k)) for k in ("k_steps", element)] == [not asked, asked]


def test_memory_of_closed_engines_can_be_given_back(fake):
    from dnlPython.engine import release_memory
    release_memory()
    base = fake.fake_used(0)
    for _ in range(2):
        with Engine(meshes.hex_block(8, 8, 8)) as e:
            e.init()
            e.ips()
    assert base < fake.fake_used(0) <= base + (256 << 20)
    release_memory()
    assert fake.fake_used(0) == base


@pytest.mark.parametrize("n", [8, 36], ids=["pool", "direct"])
def test_a_model_that_fits_only_with_the_kept_memory(fake, n):
    """Room that closed engines have left with the library is room for the next
    engine, whether it takes it from the pool or from the device."""
    d = meshes.hex_block(n, n, n)
    fake.dnl_release_memory()
    base = fake.fake_used(0)
    with Engine(d):
        need = fake.fake_used(0) - base
    fake.dnl_release_memory()
    small = [Engine(meshes.hex_block(7, 7, 7)) for _ in range(3)]
    for e in small:
        e.close()
    assert fake.fake_used(0) > base
    fake.fake_set_limit(ctypes.c_size_t(base + need))
    with Engine(d) as e:
        e.init()
    fake.dnl_release_memory()
    # and a model that does not fit is refused as before, without a trace
    fake.fake_set_limit(ctypes.c_size_t(base + need - 4096))
    with pytest.raises(_abi.EngineError, match="out of memory"):
        Engine(d)
    fake.dnl_release_memory()
    assert fake.fake_used(0) == base
