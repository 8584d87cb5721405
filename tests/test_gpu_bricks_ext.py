"""Damping and volume sweeps on the bricks (xfem_bricks_ext.cu): handles of whole
cubes too large for one thread-block cluster. Same colours, clusters and
arithmetic as the grid form, which a handle that fixes sync_mode 1 (and so builds
no bricks) runs: equal bit for bit."""
import numpy as np
import pytest

import xfem
from xfem import workloads as W

pytestmark = pytest.mark.gpu

DT = 1.0 / 1200.0
PBD = dict(pbd_damping=0.03, volume_and_time_corrected_pbd_damping=0.02,
           amortized_volume_and_time_corrected_pbd_damping=0.1)
POST, AMORTIZED = 2 << 20, 3 << 20
SWEEPS = dict(rayleigh=dict(flags=W.NH_FLAGS | POST, damping=0.005), pbd=dict(PBD),
              both=dict(PBD, flags=W.YEOH_FLAGS | AMORTIZED, damping=0.005), volume=dict(volume_passes=2),
              all=dict(PBD, flags=W.NH_FLAGS | AMORTIZED, damping=0.005, volume_passes=1))


def _settings(flags=W.NH_FLAGS, **kw):
    return xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=W.nh_compliance(1e5, 0.45),
                                 poissons_ratio=0.45, flags=flags, **kw)


def _check(meshes, settings, block, steps=(9, 1, 4)):
    """Both handles step once with plain settings: the automatic one then takes the
    bricks with the sweeps switched on."""
    plain = [_settings(ground=1, ground_normal=(0.0, 1.0, 0.0), ground_offset=-0.01, friction=0.4)] * len(meshes)
    a = xfem.Body(meshes=meshes, settings=plain, sync_mode=1, block_size=256)
    for _ in range(8):  # its launches are timed: on a busy GPU the graph of colour launches can win
        b = xfem.Body(meshes=meshes, settings=plain, block_size=block)
        b.step_frames(1, 20, DT)
        if b.info()["sync_mode"] != 2:
            break
    a.step_frames(1, 20, DT)
    for h in (a, b):
        for k, s in enumerate(settings):
            h.set_settings(s, k)
    for n in steps:
        a.step_frames(1, n, DT)
        b.step_frames(1, n, DT)
        for k in range(a.nbodies):
            assert np.array_equal(a.positions(k), b.positions(k))
            assert np.array_equal(a.velocities(k), b.velocities(k))
            assert np.array_equal(a.contacts(k), b.contacts(k))
    assert a.info()["bricks"] == 0 and b.info()["bricks"] > 1 and b.info()["sync_mode"] == 1


# ragged chunks; one brick per SM with few and with eight warps
@pytest.mark.parametrize("sweeps", sorted(SWEEPS))
@pytest.mark.parametrize("block", [128, 256])
def test_one_body(sweeps, block):
    nodes, idx = xfem.generate_tet_block(49, 33, 31, (0.05, 0.05, 0.05), 0, 0.2)
    _check([(nodes, idx, 1000.0)], [_settings(ground=1, ground_normal=(0.0, 1.0, 0.0), ground_offset=-0.01, friction=0.4,
                                              **SWEEPS[sweeps])], block)


def test_two_bricks_per_sm():
    nodes, idx = xfem.generate_tet_block(96, 64, 40, (0.05, 0.05, 0.05), 0, 0.2)
    _check([(nodes, idx, 1000.0)], [_settings(**SWEEPS["both"])], 192, (9,))


# bodies that share no vertex, each with sweeps of its own or none; vertices in
# no tet; a locked Right side
def test_bodies_and_isolated_vertices():
    meshes = []
    for n in (40, 33, 21):
        nodes, idx = xfem.generate_tet_block(n, 31, 20, (0.05, 0.05, 0.05), 0, 0.2)
        nodes = np.concatenate([np.float32([0.05, 0.5, 0.02, -0.3, 0.7, 0.1]), nodes])
        meshes.append((nodes, (idx.reshape(-1, 5) + np.uint32([0, 2, 2, 2, 2])).reshape(-1), 900.0))
    _check(meshes, [_settings(**SWEEPS["all"]), _settings(), _settings(volume_passes=3)], 192)
    _check(meshes, [_settings(**SWEEPS["rayleigh"]), _settings(**SWEEPS["pbd"]),
                    _settings(flags=W.NH_FLAGS | xfem.LOCK_RIGHT)], 224)
