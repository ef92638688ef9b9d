"""Energies and history kinetic energies, summed in a fixed order by many
blocks, against numpy's sums; node averages of every group of components."""
import numpy as np
import pytest

import helpers
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def _quads(nx, ny, precision):
    return meshes.quad_block(nx, ny, speed=60000.0, seed=5, distort=0.1, t_end=5e-6, precision=precision)


# one element's worth of lanes, a lane and a group of lanes more than 8,192
# nodes, more points than lanes (65,536)
MODELS = {"hex-8": lambda p: meshes.hex_block(2, 2, 2, speed=50000.0, seed=3, distort=0.05, t_end=5e-6, precision=p),
          "quads-8193-nodes": lambda p: _quads(2730, 2, p),
          "hex-70k-points": lambda p: meshes.taylor_3d(n_core=6, n_ring=6, n_axial=49, precision=p)}


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_energies_match_numpy(name, precision):
    from dnlPython.engine import Engine
    d = MODELS[name](precision)
    g = np.random.default_rng(1)
    with Engine([d, d.copy(t_end=2e-6)]) as e:
        e.init()
        s = e.ips()
        s[_abi.IP_EINT:_abi.IP_EINEL + 1] = g.uniform(0.5, 1.5, (2, e.n_ips)).astype(np.float32)
        e.set_ips(s)
        v = g.standard_normal((e.n_nodes, 3))
        e.set_nodes(_abi.NODE_SPEED, v)
        e.set_items([(_abi.ITEM_KINETIC, _abi.NODE_SPEED, k) for k in (0, 1)])
        kin = e.gather_items()
        for k in (0, 1):
            n0, e0, q0 = e.offsets(k)
            n1, q1 = (e.offsets(1)[0], e.offsets(1)[2]) if k == 0 else (e.n_nodes, e.n_ips)
            m = e.nodes(_abi.NODE_MASS)[n0:n1, 0]
            w = d.materials[0]["density"] * e.ips()[_abi.IP_DETJ0, q0:q1]
            want = [np.sum(0.5 * m * (v[n0:n1] ** 2).sum(1)), np.sum(w * s[_abi.IP_EINT, q0:q1]),
                    np.sum(w * s[_abi.IP_EINEL, q0:q1])]
            # positive terms: the sums' relative rounding is below (additions in a row) x 2^-53
            assert np.allclose(e.energies(k), want, rtol=1e-13, atol=0)
            assert kin[k] == e.energies(k)[0]


@pytest.mark.parametrize("n", [1, 4, 5, 33])
def test_node_averages_of_any_number_of_components(n):
    """Groups of components share a thread: every count gives what a call per component gives."""
    from dnlPython.engine import Engine
    d = helpers.case_hex_small(_abi.PREC_MIXED)
    comps = ([_abi.NODE_AVG_VON_MISES] + list(range(_abi.IP_NCOMP)) * 2)[:n]
    with Engine(d) as e:
        e.init()
        e.run(max_incs=15)
        got = e.node_averages(comps)
        for k, c in enumerate(comps):
            assert np.array_equal(got[k], e.node_averages([c])[0])
