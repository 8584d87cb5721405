"""The one-cluster form of the persistent tet kernel (xfem_cluster.cu): handles
small enough run sync_mode 1 as one thread-block cluster with the vertices in
its distributed shared memory. Same colours, chunks and arithmetic as the grid
form, which handles that keep multipliers still take: equal bit for bit."""
import numpy as np
import pytest

import xfem
from xfem import workloads as W

pytestmark = pytest.mark.gpu

DT = 1.0 / 1200.0
DAMPED = dict(damping=0.005, pbd_damping=0.03, volume_and_time_corrected_pbd_damping=0.02,
              amortized_volume_and_time_corrected_pbd_damping=0.1)


def _settings(flags=W.NH_FLAGS, **kw):
    return xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=W.nh_compliance(1e5, 0.45),
                                 poissons_ratio=0.45, flags=flags, **kw)


def _pair(meshes, settings, **opts):
    a = xfem.Body(meshes=meshes, settings=settings, sync_mode=1, **opts)
    b = xfem.Body(meshes=meshes, settings=settings, sync_mode=1, keep_lambdas=True, **opts)
    return a, b


def _same(a, b, steps=(13, 1, 4)):
    for n in steps:
        a.step_frames(1, n, DT)
        b.step_frames(1, n, DT)
        for k in range(a.nbodies):
            assert np.array_equal(a.positions(k), b.positions(k))
            assert np.array_equal(a.velocities(k), b.velocities(k))
            assert np.array_equal(a.contacts(k), b.contacts(k))


# one cube (one colour); one chunk per colour; two blocks, ragged chunks; the
# largest bodies of one round at 64 and at 256 threads (32 and 128 chunks of a
# colour) and one larger than the latter, which keeps the grid
@pytest.mark.parametrize("dims,block", [((1, 1, 1), 64), ((8, 2, 2), 128), ((9, 7, 5), 64), ((17, 12, 11), 128),
                                        ((32, 16, 16), 64), ((64, 32, 16), 256), ((66, 32, 16), 256)])
def test_cube_bodies(dims, block):
    nodes, idx = xfem.generate_tet_block(*dims, (0.1, 0.1, 0.1), 0, 0.2)
    _same(*_pair([(nodes, idx, 1000.0)], [_settings()], block_size=block))


# one tet per lane (more colours than the descriptors kept in shared memory),
# mirrored cubes (clusters of other shapes), vertices in no tet, several bodies
@pytest.mark.parametrize("mesh", ["one_tet", "mirrored", "isolated", "batch"])
@pytest.mark.parametrize("sweeps", ["plain", "damped", "volume"])
def test_other_chunks_and_sweeps(mesh, sweeps):
    kw = dict(plain={}, damped=dict(DAMPED, flags=W.YEOH_FLAGS | (3 << 20)), volume=dict(volume_passes=2))[sweeps]
    s = _settings(ground=1, ground_normal=(0.0, 1.0, 0.0), ground_offset=-0.31, friction=0.4, **kw)
    nodes, idx = xfem.generate_tet_block(7, 6, 5, (0.1, 0.1, 0.1), 1 if mesh == "mirrored" else 0, 0.3)
    if mesh == "isolated":
        nodes = np.concatenate([np.float32([0.05, 0.5, 0.02, -0.3, 0.7, 0.1]), nodes])
        idx = (idx.reshape(-1, 5) + np.uint32([0, 2, 2, 2, 2])).reshape(-1)
    meshes = [(nodes, idx, 1000.0)]
    if mesh == "batch":
        meshes = [xfem.generate_tet_block(n, 4, 3, (0.1, 0.1, 0.1), n % 2, 0.2) + (900.0,) for n in (2, 5, 9)]
    a, b = _pair(meshes, [s] * len(meshes), block_size=128, cluster_mode=1 if mesh == "one_tet" else 0)
    _same(a, b, (11, 9))


def test_switching_damping_on_and_off():
    nodes, idx = xfem.generate_tet_block(9, 7, 5, (0.1, 0.1, 0.1), 0, 0.2)
    a, b = _pair([(nodes, idx, 1000.0)], [_settings()], block_size=128)
    for flags, kw in ((W.NH_FLAGS | (2 << 20), DAMPED), (W.NH_FLAGS, {})):
        _same(a, b, (3,))
        for h in (a, b):
            h.set_settings(_settings(flags=flags, **kw))
        _same(a, b, (5,))


@pytest.mark.parametrize("dims", [(8, 2, 2), (20, 9, 9)])
def test_recording_forward_is_the_plain_one(dims):
    nodes, idx = xfem.generate_tet_block(*dims, (0.1, 0.1, 0.1), 0, 0.2)
    a, b = _pair([(nodes, idx, 1000.0)], [_settings()], block_size=128)
    tips = np.uint32([0, nodes.size // 3 - 1])
    traj = a.adjoint_forward(12, DT, tips, 5)
    b.step_frames(1, 12, DT)
    assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities(), b.velocities())
    assert np.array_equal(traj[-1], b.positions()[tips])


# the reverse as one cluster: one block; one, two and three rounds of chunks per
# block; one more than that (the grid form); two bodies; checkpointed segments
@pytest.mark.parametrize("dims,every", [([(8, 2, 2)], 0), ([(8, 2, 2)], 3), ([(20, 9, 9)], 4), ([(32, 16, 12)], 0),
                                        ([(32, 20, 16)], 0), ([(32, 21, 20)], 0), ([(5, 4, 3), (9, 2, 7)], 5)])
@pytest.mark.parametrize("ground", [0, 1])
def test_reverse_matches_the_one_lane_form(dims, every, ground, monkeypatch):
    nsub = 7
    s = _settings(ground=ground, ground_normal=(0.0, 1.0, 0.0), ground_offset=-0.5 * 0.1 * dims[0][1] + 0.01, friction=0.4)
    rng = np.random.default_rng(3)
    meshes = [xfem.generate_tet_block(*d, (0.1, 0.1, 0.1), 0, 0.2) + (1000.0,) for d in dims]
    b = xfem.Body(meshes=meshes, settings=[s] * len(meshes))
    nv = sum(c[0] for c in b.counts)
    tips = np.uint32([0, nv // 2, nv - 1])
    b.adjoint_forward(nsub, DT, tips, every)
    g = rng.standard_normal((nsub, 3, 3)).astype(np.float32)
    gx, gv = (rng.standard_normal((nv, 3)).astype(np.float32) for _ in range(2))
    got = b.adjoint_backward(g, gx, gv)
    monkeypatch.setenv("XFEM_REVERSE_FORM", "lane")
    for x, y in zip(got, b.adjoint_backward(g, gx, gv)):
        assert np.array_equal(x, y) and np.abs(x).max() > 0
