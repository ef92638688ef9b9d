"""Records of small models (increments in one cooperative launch): the first
block reads a record's items while the other blocks wait.  What they would
change if they went on is asked for: the densities of the last tiles with the
time step due at every increment (and the kinetic energies, which are read
before them), and u, v and a of more imposed-speed nodes than the first block
prepares (128)."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu

KINETIC = [(_abi.ITEM_KINETIC, f, 0) for f in (_abi.NODE_SPEED, _abi.NODE_SPEED_PREV)]


def _free(precision, **kw):
    """422 tiles, 13,720 nodes, no imposed speed; points of every 16th tile and the last."""
    d = meshes.quad_block(97, 139, size=(1.0, 139 / 97), speed=60000.0, seed=5, distort=0.1, t_end=5e-6, ts_freq=1,
                          precision=precision, **kw)
    return d, KINETIC + [(_abi.ITEM_POINT, 0, q) for q in [*range(d.n_ips - 1, 0, -16 * 128), 0]]


def _pulled(precision):
    """2,880 hexahedra (180 tiles), 169 nodes pulled; the ramp ends within the run."""
    d = meshes.plate_necking(nx=12, nz=12, ny=20, width=1.0, length=3.0, speed=50000.0, elongation=0.5,
                             ramp_frac=0.02, ts_freq=1, precision=precision)
    end = np.flatnonzero(d.bc_code[:, 1] == _abi.BC_SPEED)
    assert end.size == 169
    return d, KINETIC + [(_abi.ITEM_NODE, f, int(i)) for f in (_abi.NODE_U, _abi.NODE_SPEED, _abi.NODE_ACCEL)
                         for i in end] + [(_abi.ITEM_POINT, 0, d.n_ips - 1)]


def _free_power(precision):
    d, items = _free(precision)
    return d.copy(ts_method=_abi.TS_POWER_ITERATION), items


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("model", [_free, _pulled, _free_power], ids=["free", "pulled", "free-power"])
def test_records_equal_stopping_at_each_increment(model, precision):
    """Every value of every record, bit for bit, as a run that stops after each increment gathers it."""
    from dnlPython.engine import Engine
    d, items = model(precision)
    incs = 6 if model is _free_power else 30
    with Engine(d) as e:
        e.init()
        e.set_items(items)
        e.set_history([(0.0, 0.0, 0.0)], capacity=64)
        e.run(max_incs=incs)
        assert e.launch_count() <= 2  # the limits and one launch
        rec = e.history_records()
    assert len(rec) == incs
    with Engine(d) as e:
        e.init()
        e.set_items(items)
        for k in range(incs):
            e.run(max_incs=1)
            c = e.control()
            assert rec[k][:3] == (c["time"], c["increment"], c["last_time_step"])
            assert np.array_equal(rec[k][4], e.gather_items()), k
