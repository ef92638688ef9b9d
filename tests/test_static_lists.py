"""Force assembly of dnl_element_pass_static: nodes with as many elements as a
list holds, with fewer, and with more (assembled through lists of any length)."""
import numpy as np
import pytest

import helpers
import test_zz_no_alloc as base
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def _fan(n, layers):
    """n quads around one node in the (x, y) plane (each: the centre, a spoke's
    end, a rim corner, the next spoke's end); layers > 0: extruded to hexahedra."""
    a = 2.0 * np.pi * np.arange(n) / n
    mid = a + np.pi / n
    pts = np.concatenate([[[5.0, 0.0]], np.stack([5.0 + np.cos(a), np.sin(a)], 1),
                          np.stack([5.0 + 1.3 * np.cos(mid), 1.3 * np.sin(mid)], 1)])
    quads = np.array([[0, 1 + k, 1 + n + k, 1 + (k + 1) % n] for k in range(n)])
    if layers == 0:
        coords = np.zeros((len(pts), 3))
        coords[:, :2] = pts
        return _abi.ModelDesc(_abi.ELQUA4NAX, coords, quads, [meshes.COPPER], t_end=1e-5)
    coords = np.zeros(((layers + 1) * len(pts), 3))
    conn = []
    for k in range(layers + 1):
        coords[k * len(pts):(k + 1) * len(pts), :2] = pts
        coords[k * len(pts):(k + 1) * len(pts), 2] = 0.8 * k
        if k < layers:
            conn.append(np.concatenate([quads + k * len(pts), quads + (k + 1) * len(pts)], 1))
    return _abi.ModelDesc(_abi.ELHEX8N3D, coords, np.concatenate(conn), [meshes.COPPER], t_end=1e-5)


@pytest.mark.parametrize("n,layers", [(4, 0), (5, 0), (4, 3), (5, 3), (11, 2)])
def test_static_pass_assembles_nodes_of_any_valence(n, layers):
    desc = _fan(n, layers)
    u = helpers.random_increment(desc, seed=3, strain=3e-3)
    dt = 9e-9
    from oracle import OracleModel
    with OracleModel(desc) as o:
        o.init()
        ips = helpers.random_point_state(desc, o.ips(), seed=4, stress_scale=250.0)
    x, ip_ref, f_ref = base._reference_pass(desc, ips, u, dt)
    for _ in range(2):
        ip_s, f_s = base._static_pass(desc, x, u, ips, dt)
        assert helpers.field_errors(ip_s, ip_ref).max() < 1e-9
        assert helpers.rel_err(f_s, f_ref) < 1e-9
