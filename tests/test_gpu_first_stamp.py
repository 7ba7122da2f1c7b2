"""The first body call of a world clears its claims before it uses them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(64, 64), (8192, 4096)])
def test_first_stamp_of_a_world(fse, w, h):
    """Memory that another world's claims lay in is given out again: every tile of a box in
    free cells must be placed, in each of a few fresh worlds."""
    n = 32
    for k in range(4):
        with fse.World(w, h, seed=k, particle_capacity=1024) as world:
            b = np.zeros(n, fse.BODY_DTYPE)
            b["w"] = b["h"] = 8
            b["x"], b["y"] = (np.arange(n) % 8) * 8, (np.arange(n) // 8) * 8
            b["x"] += w - 64
            b["y"] += h - 64
            b["cos_a"] = 1.0
            b["id"] = fse.material_find("GENERIC_OBJECT")
            world.object_stamp(b)
            assert (b["n_placed"] == 64).all()
            assert world.object_readback(b) == 64 * n
