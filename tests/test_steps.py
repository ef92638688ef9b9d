"""Increments of small models in one cooperative launch (k_steps) against the
same increments kernel by kernel (a variant asked for with set_variant runs so)."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def engine(desc):
    from dnlPython.engine import Engine
    return Engine(desc)


def _quads(nx, ny, precision, **kw):
    return meshes.quad_block(nx, ny, size=(1.0, ny / nx), speed=60000.0, seed=5, distort=0.1, t_end=5e-6,
                             precision=precision, **kw)


MODELS = {
    # fewer points than a tile, a tile and a remainder, several tiles; imposed
    # speeds with a time function; the most tiles a register budget holds
    # (148 x 2 and one more, FP64) and one more than all (kernel by kernel)
    "hex-8": lambda p: meshes.hex_block(2, 2, 2, speed=50000.0, seed=3, distort=0.05, t_end=5e-6, precision=p),
    "hex-17": lambda p: meshes.hex_block(17, 1, 1, size=(17.0, 1.0, 1.0), speed=60000.0, seed=2, distort=0.05,
                                         t_end=5e-6, precision=p, ts_freq=3),
    "hex-speed": lambda p: helpers.case_hex_speed(p),
    "axi": lambda p: meshes.taylor_axi(nr=5, nz=23, precision=p, ts_freq=1),
    "plane": lambda p: _quads(13, 29, p),
    "bar-297-tiles": lambda p: meshes.taylor_3d(n_core=4, n_ring=4, n_axial=59, length=12.0, precision=p),
    "plane-large": lambda p: _quads(120, 161, p),
}


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_steps_equal_kernel_by_kernel(name, precision):
    """Same increments, times and (FP64: to the rounding of fused multiply-adds,
    amplified over 60 increments; mixed: one material and variant 0, bit for
    bit) the same state, whatever pieces the run is cut into."""
    d = MODELS[name](precision)
    out = []
    for forced, pieces in ((True, [60]), (False, [60]), (False, [1, 7, 30, 22])):
        with engine(d) as e:
            e.init()
            if forced:
                e.set_variant(0)
            for n in pieces:
                e.run(max_incs=n)
            c = e.control()
            out.append((e.nodes(_abi.NODE_COORDS), e.nodes(_abi.NODE_SPEED), e.ips(), c["increment"], c["time"],
                        c["status"]))
    ref, one, cut = out
    assert ref[3] == one[3] == cut[3] and ref[5] == one[5] == cut[5] == 0
    for a, b in zip(one, cut):
        assert np.array_equal(a, b)
    if precision == _abi.PREC_MIXED:
        for a, b in zip(ref, one):
            assert np.array_equal(a, b)
    else:
        assert abs(ref[4] - one[4]) <= 1e-12 * ref[4]
        assert helpers.rel_err(one[0], ref[0]) < 1e-12 and helpers.rel_err(one[1], ref[1]) < 1e-10
        assert helpers.field_errors(one[2], ref[2]).max() < 1e-8


def test_steps_stop_at_a_failed_element_and_keep_timings():
    """An inverted element stops the launch with its status at the same
    increment as kernel by kernel; the phase times of a timed run add up to
    no more than the run's."""
    d = helpers.case_hex_small()
    got = []
    for forced in (True, False):
        with engine(d) as e:
            e.init()
            if forced:
                e.set_variant(0)
            x = e.nodes(_abi.NODE_COORDS)
            k = d.conn[0]
            x[k[6]] = x[k[0]] - (x[k[6]] - x[k[0]])
            e.set_nodes(_abi.NODE_COORDS, x)
            with pytest.raises(_abi.EngineError):
                e.run(max_incs=5)
            c = e.control()
            # (several elements share the node: which of them is reported is not defined)
            got.append((c["status"], c["increment"], c["time"]))
    assert got[0] == got[1] and got[0][0] == _abi.DNL_ERR_NEG_JACOBIAN
    with engine(d) as e:
        e.init()
        e.set_timing(True)
        e.run(max_incs=40)
        t = e.timings()
        assert min(t.values()) > 0.0
        assert t["element_ms"] + t["nodal_ms"] + t["timestep_ms"] <= t["run_ms"]


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["axi", "hex-17", "hex-speed", "plane", "bar-297-tiles"])
def test_power_iteration_in_steps(name, precision):
    """The power-iteration time step inside the launch: same increments, and
    time steps, iteration by iteration the sums of its own kernel; a run cut
    into pieces goes on from the kept vector."""
    d = MODELS[name](precision).copy(ts_method=_abi.TS_POWER_ITERATION, ts_freq=2)
    out = []
    for forced, pieces in ((True, [24]), (False, [24]), (False, [1, 6, 17])):
        with engine(d) as e:
            e.init()
            if forced:
                e.set_variant(0)
            for n in pieces:
                e.run(max_incs=n)
            c = e.control()
            out.append((e.nodes(_abi.NODE_COORDS), e.ips(), c["increment"], c["time"], c["time_step"], c["status"]))
    ref, one, cut = out
    assert ref[2] == one[2] == cut[2] and ref[5] == one[5] == cut[5] == 0
    assert np.array_equal(one[0], cut[0]) and np.array_equal(one[1], cut[1]) and one[3:5] == cut[3:5]
    assert abs(one[4] - ref[4]) <= 1e-11 * ref[4]
    # the time steps differ by rounding at most, so the states do as two FP64 or
    # two mixed runs a rounding apart
    assert helpers.rel_err(one[0], ref[0]) < (1e-12 if precision == _abi.PREC_FP64 else 1e-7)
    assert helpers.field_errors(one[1], ref[1]).max() < (1e-8 if precision == _abi.PREC_FP64 else 1e-3)
