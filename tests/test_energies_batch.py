"""Energies of a batch of more instances than a grid has rows (65,535)."""
import numpy as np
import pytest

import helpers  # noqa: F401
from dnlPython import _abi, meshes

pytestmark = pytest.mark.gpu


def test_energies_of_many_instances():
    from dnlPython.engine import Engine
    d = meshes.hex_block(1, 1, 1, size=(0.5, 0.7, 0.9))
    n = 65_600
    g = np.random.default_rng(3)
    with Engine([d] * n) as e:
        e.init()
        v = g.standard_normal((e.n_nodes, 3))
        e.set_nodes(_abi.NODE_SPEED, v)
        m = e.nodes(_abi.NODE_MASS)[:, 0]
        kinetic = (0.5 * m * (v ** 2).sum(1)).reshape(n, 8).sum(1)
        items = [0, 1, 65_535, 65_536, n - 1]
        e.set_items([(_abi.ITEM_KINETIC, _abi.NODE_SPEED, k) for k in items])
        got = e.gather_items()
        # (8 positive terms: a few roundings of 2^-53)
        assert np.allclose(got, kinetic[items], rtol=2e-15, atol=0)
        assert [e.energies(k)[0] for k in items] == list(got)
