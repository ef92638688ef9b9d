"""The element pass with a tile's point state by one bulk copy (variant 0 of the
mixed path) against the staged pass (variant 5): models of less than a tile, a
tile and a remainder, many tiles, and batches whose tiles hold points of two
instances and of which some stop early."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def _block(n, seed, t_end=5e-6):
    return meshes.hex_block(n, 1, 1, size=(float(n), 1.0, 1.0), speed=50000.0, seed=seed, distort=0.05, t_end=t_end,
                            precision=_abi.PREC_MIXED, ts_freq=3)


MODELS = {"8": lambda: [meshes.hex_block(2, 2, 2, speed=50000.0, seed=3, distort=0.05, t_end=5e-6,
                                         precision=_abi.PREC_MIXED)],
          "16": lambda: [_block(16, 2)], "17": lambda: [_block(17, 2)],
          "bar": lambda: [meshes.taylor_3d(n_core=4, n_ring=4, n_axial=59, length=12.0)],
          "batch": lambda: [_block(16, 4), _block(5, 5, t_end=1e-6), _block(23, 6), _block(3, 7), _block(17, 8, 2e-6)]}


def _run(descs, variant):
    from dnlPython.engine import Engine
    with Engine(descs) as e:
        e.init()
        e.set_variant(variant)
        for n in (20, 1, 19):
            e.run(max_incs=n, check=False)
        c = [e.control(k) for k in range(e.n_instances)]
        return e.nodes(_abi.NODE_COORDS), e.ips(), [(x["increment"], x["status"]) for x in c]


@pytest.mark.parametrize("name", sorted(MODELS))
def test_once_equals_staged(name):
    descs = MODELS[name]()
    a, b = _run(descs, 0), _run(descs, 5)
    # (the three-element instance of the batch inverts in the C restatement too,
    # at its ninth increment: it stops alone)
    assert a[2] == b[2]
    assert [s for _, s in a[2]] == ([0, 0, 0, _abi.DNL_ERR_NEG_JACOBIAN, 0] if name == "batch" else [0])
    # the bounds of the variants among each other (test_gpu_parity.py)
    assert helpers.rel_err(a[0], b[0]) < 1e-7
    assert helpers.field_errors(a[1], b[1]).max() < 1e-3
    again = _run(descs, 0)
    assert np.array_equal(a[0], again[0]) and np.array_equal(a[1], again[1])
