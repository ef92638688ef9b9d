"""Cooperative increments (k_steps) of models of two materials, whose builds read
the law's constants from memory, at both register budgets of either precision
(296 and 444 tiles of 128 points in FP64, 444 and 592 mixed, on 148 SMs) and with
both time steps, against the same increments kernel by kernel; and the second
budget of the mixed builds of one material."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def _two(d):
    """Two materials in turn: another yield stress, hardening exponent and density."""
    a = d.materials[0]
    b = dict(a, A=1.3 * a["A"], n=0.8 * a["n"], density=1.1 * a["density"])
    return d.copy(materials=[a, b], elem_mat=(np.arange(d.n_elems) % 3 == 1).astype(np.int32))


def _quads(nx, ny, precision, elem_type):
    return meshes.quad_block(nx, ny, size=(1.0, ny / nx), speed=60000.0, seed=5, distort=0.1, t_end=5e-6,
                             precision=precision, elem_type=elem_type)


MODELS = {
    "hex-17": lambda p: meshes.hex_block(17, 1, 1, size=(17.0, 1.0, 1.0), speed=60000.0, seed=2, distort=0.05,
                                         t_end=5e-6, precision=p, ts_freq=3),
    "hex-320-tiles": lambda p: meshes.hex_block(16, 20, 16, size=(1.6, 2.0, 1.6), speed=60000.0, seed=2, distort=0.05,
                                                t_end=5e-6, precision=p),
    "hex-500-tiles": lambda p: meshes.hex_block(20, 20, 20, size=(2.0, 2.0, 2.0), speed=60000.0, seed=2, distort=0.05,
                                                t_end=5e-6, precision=p),
    "axi-12-tiles": lambda p: _quads(13, 29, p, _abi.ELQUA4NAX),
    "plane-318-tiles": lambda p: _quads(90, 113, p, _abi.ELQUA4N2D),
    "plane-504-tiles": lambda p: _quads(115, 140, p, _abi.ELQUA4N2D),
}
TILES = {_abi.PREC_FP64: 444, _abi.PREC_MIXED: 592}


def _run(d, incs, forced):
    from dnlPython.engine import Engine
    with Engine(d) as e:
        e.init()
        if forced:
            e.set_variant(0)
        e.run(max_incs=incs)
        assert forced or e.launch_count() == 2  # the limits and one launch
        c = e.control()
        assert c["status"] == 0
        return e.nodes(_abi.NODE_COORDS), e.nodes(_abi.NODE_SPEED), e.ips(), c["increment"], c["time"], c["time_step"]


def _cases():
    for p in (_abi.PREC_FP64, _abi.PREC_MIXED):
        for name in sorted(MODELS):
            tiles = int(name.split("-")[1]) if name.endswith("tiles") else 2
            if tiles > TILES[p]:
                continue
            for power in (False, True):
                yield pytest.param(name, p, True, power)
                if tiles > 444:
                    yield pytest.param(name, p, False, power)


@pytest.mark.parametrize("name,precision,two,power", list(_cases()))
def test_steps_equal_kernel_by_kernel(name, precision, two, power):
    """The bounds of test_steps.py: the mixed builds bit for bit with the Courant
    time step, to rounding (FP64) or as two mixed runs a rounding apart with the
    power iteration's."""
    d = MODELS[name](precision)
    if two:
        d = _two(d)
    if power:
        d = d.copy(ts_method=_abi.TS_POWER_ITERATION, ts_freq=2)
    incs = 12 if power else 25
    ref, one = _run(d, incs, True), _run(d, incs, False)
    assert ref[3] == one[3] == incs
    if precision == _abi.PREC_MIXED and not power:
        for a, b in zip(ref, one):
            assert np.array_equal(a, b)
        return
    assert abs(one[4] - ref[4]) <= 1e-11 * ref[4] and abs(one[5] - ref[5]) <= 1e-11 * ref[5]
    fp64 = precision == _abi.PREC_FP64
    assert helpers.rel_err(one[0], ref[0]) < (1e-12 if fp64 else 1e-7)
    assert not fp64 or helpers.rel_err(one[1], ref[1]) < 1e-10
    assert helpers.field_errors(one[2], ref[2]).max() < (1e-8 if fp64 else 1e-3)
