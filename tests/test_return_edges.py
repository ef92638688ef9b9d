"""Returns whose Johnson-Cook law has arguments outside the normal numbers, FP64
path against the C restatement (libm's pow and log): plastic strains below the
normal numbers, a material that does not soften (infinite melting temperature)
with a small exponent, and inputs for which the return does not converge."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi

pytestmark = pytest.mark.gpu
DT = 9e-9


def _state(kind, change):
    """Model, displacement increment and point state of one pass."""
    d = helpers.case_hex_small() if kind == "hex" else helpers.case_axi_small()
    u = helpers.random_increment(d, seed=7, strain=2e-3)
    mat = dict(d.materials[0], **({"Tm": np.inf, "m": 0.03} if change == "no-melting" else
                                  {"depsp0": 0.0} if change == "no-rate" else {}))
    d = d.copy(materials=[mat])
    from oracle import OracleModel
    with OracleModel(d) as o:
        o.init()
        ips = helpers.random_point_state(d, o.ips(), seed=8, stress_scale=250.0)
    # every point yields: a small yield stress, whatever its plastic strain
    ips[_abi.IP_YIELD] = 50.0
    if change == "subnormal":
        ips[_abi.IP_EPSP, ::3] = 10.0 ** np.random.default_rng(4).uniform(-322, -309, ips[0, ::3].size)
        ips[_abi.IP_GAMMA, ::3] = 0.0
    if change == "infinite":
        ips[_abi.IP_EPSP, 5] = np.inf
    return d, u, ips


def _pass(m, u, ips):
    m.init()
    m.set_ips(ips)
    m.set_nodes(_abi.NODE_U, u)
    m.element_pass(DT)
    return m.ips(), m.nodes(_abi.NODE_FORCE)


@pytest.mark.parametrize("kind", ["hex", "axi"])
@pytest.mark.parametrize("change", ["none", "subnormal", "no-melting"])
def test_returns_at_the_edges_of_the_law(kind, change):
    from dnlPython.engine import Engine
    from oracle import OracleModel
    d, u, ips = _state(kind, change)
    with OracleModel(d) as o, Engine(d) as e:
        want, f = _pass(o, u, ips)
        got, g = _pass(e, u, ips)
    assert (want[_abi.IP_YIELD] != 50.0).mean() > 0.5
    assert helpers.field_errors(got, want).max() < 1e-9
    assert helpers.rel_err(g, f) < 1e-9


@pytest.mark.parametrize("kind", ["hex", "axi"])
@pytest.mark.parametrize("change", ["infinite", "no-rate"])
def test_returns_without_a_finite_law_do_not_converge(kind, change):
    from dnlPython.engine import Engine
    from oracle import OracleModel
    d, u, ips = _state(kind, change)
    with OracleModel(d) as o:
        with pytest.raises(RuntimeError, match="element_pass failed"):
            _pass(o, u, ips)
    with Engine(d) as e:
        with pytest.raises(_abi.EngineError) as x:
            _pass(e, u, ips)
        assert x.value.code == _abi.DNL_ERR_NEWTON
