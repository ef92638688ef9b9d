"""Device memory that closed engines leave with the library goes back to the device on request."""
import pytest

import helpers  # noqa: F401
from dnlPython import meshes

pytestmark = pytest.mark.gpu


def test_kept_memory_goes_back_to_the_device():
    import torch
    from dnlPython.engine import Engine, release_memory

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    d = meshes.hex_block(24, 24, 24)
    with Engine(d) as e:  # loads the kernels
        e.init()
    release_memory()
    before = free()
    with Engine(d) as e:
        e.init()
    kept = before - free()
    assert 16 << 20 < kept <= 256 << 20  # (the engine holds some 45 MB)
    release_memory()
    assert before - free() <= 2 << 20
    with Engine(d) as e:
        e.init()
        e.run(max_incs=3)
