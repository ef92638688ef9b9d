"""Device memory kept from engine to engine: engines created, run and closed in
any order, from several threads at once, and a closed engine's memory reused by
another model, give what they give alone."""
import threading

import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def _solve(d):
    from dnlPython.engine import Engine
    with Engine(d) as e:
        e.init()
        e.set_items([(_abi.ITEM_KINETIC, _abi.NODE_SPEED, 0), (_abi.ITEM_POINT, 0, 3)])
        e.run(max_incs=20)
        return e.nodes(_abi.NODE_COORDS), e.ips(), e.gather_items(), e.node_averages([_abi.IP_EPSP])


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_memory_of_closed_engines_is_reused_cleanly():
    descs = [helpers.case_hex_small(), helpers.case_axi_small(),
             helpers.case_hex_speed().copy(ts_method=_abi.TS_POWER_ITERATION, ts_freq=2),
             meshes.taylor_3d(n_core=4, n_ring=4, n_axial=30, precision=_abi.PREC_MIXED)]
    want = [_solve(d) for d in descs]
    for order in ([3, 0, 2, 1], [1, 3, 0, 2], [2, 2, 3, 1]):
        for k in order:
            assert _equal(_solve(descs[k]), want[k]), k


def test_engines_of_several_threads():
    descs = [helpers.case_hex_small(), helpers.case_axi_small(), helpers.case_hex_speed()]
    want = [_solve(d) for d in descs]
    bad = []

    def work(k):
        try:
            for _ in range(6):
                if not _equal(_solve(descs[k]), want[k]):
                    bad.append(k)
        except Exception as e:  # noqa: BLE001
            bad.append((k, e))

    threads = [threading.Thread(target=work, args=(k % len(descs),)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
