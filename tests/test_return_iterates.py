"""The FP64 return evaluates the Johnson-Cook law by its own straight-line
logarithm and exponential (JC::eval64): starts below, near and far above the
root, plastic strains over six decades and first yield, cold points, points at
the reference temperature and about to melt, against the C restatement (libm's
pow and log)."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["hex", "axi"])
@pytest.mark.parametrize("start", [0.0, 1e-3, 0.5, 0.86, 0.88, 0.98, 1.0, 1.02, 1.15, 4.0])
def test_returns_from_near_and_far_starts(kind, start):
    from dnlPython.engine import Engine
    from oracle import OracleModel
    d = helpers.case_hex_small() if kind == "hex" else helpers.case_axi_small()
    u = helpers.random_increment(d, seed=7, strain=2e-3)
    dt = 9e-9
    with OracleModel(d) as o:
        o.init()
        ips = helpers.random_point_state(d, o.ips(), seed=8, stress_scale=250.0)
        g = np.random.default_rng(9)
        m = d.materials[0]
        n = d.n_ips
        ips[_abi.IP_EPSP] = 10.0 ** g.uniform(-6, 0, n)
        ips[_abi.IP_T] = g.choice([m["Tref"] - 5.0, m["Tref"], m["Tref"] + 0.5, 600.0, m["Tm"] - 0.1, m["Tm"] - 30.0], n)
        ips[_abi.IP_EPSP, ::17] = 0.0
        # the converged multipliers of this pass as the next one's starts, scaled
        o.set_ips(ips)
        o.set_nodes(_abi.NODE_U, u)
        o.element_pass(dt)
        ips[_abi.IP_GAMMA] = start * o.ips()[_abi.IP_GAMMA]
        o.set_ips(ips)
        o.set_nodes(_abi.NODE_U, u)
        o.element_pass(dt)
        want, f = o.ips(), o.nodes(_abi.NODE_FORCE)
        x = o.nodes(_abi.NODE_COORDS)
    assert (want[_abi.IP_GAMMA_CUM] > ips[_abi.IP_GAMMA_CUM]).mean() > 0.2
    with Engine(d) as e:
        e.init()
        e.set_nodes(_abi.NODE_COORDS, x)
        e.set_ips(ips)
        e.set_nodes(_abi.NODE_U, u)
        e.element_pass(dt)
        got = e.ips()
        # a point that melts returns to a zero deviator: its plastic strain, gamma
        # over what is left of it times what is left of it, is rounding in both codes
        molten = want[_abi.IP_YIELD] == 0.0
        got[12:18, molten] = want[12:18, molten]
        assert helpers.field_errors(got, want).max() < 1e-9
        assert helpers.rel_err(e.nodes(_abi.NODE_FORCE), f) < 1e-9
