"""How the clusters are divided into bricks (split_bricks in xfem_api.cpp): parts
across a body's longest side, or Morton runs. The results do not depend on it:
each split equals the persistent form bit for bit."""
import numpy as np
import pytest

import xfem
from xfem import workloads as W

pytestmark = pytest.mark.gpu

DT = 1.0 / 1200.0


def _check(meshes, block, bricks=0):
    s = xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=W.nh_compliance(1e5, 0.45), poissons_ratio=0.45,
                              flags=W.NH_FLAGS)
    a = xfem.Body(meshes=meshes, settings=[s] * len(meshes), sync_mode=1, block_size=256)
    b = xfem.Body(meshes=meshes, settings=[s] * len(meshes), sync_mode=4, block_size=block, bricks=bricks)
    for h in (a, b):
        h.step_frames(1, 7, DT)
        h.step_frames(1, 2, DT)
    for k in range(a.nbodies):
        assert np.array_equal(a.positions(k), b.positions(k))
        assert np.array_equal(a.velocities(k), b.velocities(k))
    assert b.info()["sync_mode"] == 4


# one column of cubes, a plate, ragged sides; a body that two bricks per SM take
# in runs, and one whose slabs beyond a power of two need the parts
@pytest.mark.parametrize("dims,block", [((1, 1, 3000), 128), ((90, 60, 1), 256), ((37, 29, 31), 256), ((96, 64, 40), 192),
                                        ((127, 65, 33), 192)])
def test_one_body(dims, block):
    nodes, idx = xfem.generate_tet_block(*dims, (0.05, 0.05, 0.05), 0, 0.2)
    _check([(nodes, idx, 1000.0)], block)


# bodies at the same place, smaller than a brick and of several bricks; vertices
# of one layer apart by rounding only; a requested number of bricks
@pytest.mark.parametrize("bricks", [0, 5])
def test_bodies(bricks):
    rng = np.random.default_rng(3)
    meshes = []
    for d in ((3, 3, 3), (25, 11, 13), (2, 2, 2), (12, 12, 12), (9, 40, 5)):
        nodes, idx = xfem.generate_tet_block(*d, (0.05, 0.05, 0.05), 0, 0.2)
        meshes.append(((nodes * (1.0 + 1e-6 * rng.standard_normal(nodes.size))).astype(np.float32), idx, 900.0))
    _check(meshes, 256, bricks)
