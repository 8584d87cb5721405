"""Which form each kind of call runs in (xfem_get_launch): the forms give equal
results, so that a comparison of two of them holds just as well when both handles
took the same one."""
import numpy as np
import pytest

import xfem
from xfem import workloads as W

pytestmark = pytest.mark.gpu

DT = 1.0 / 1200.0
PBD = dict(pbd_damping=0.03, volume_and_time_corrected_pbd_damping=0.02,
           amortized_volume_and_time_corrected_pbd_damping=0.1)
DAMPED = dict(PBD, flags=W.NH_FLAGS | (2 << 20), damping=0.005)
SWEEPS = dict(rayleigh=dict(flags=W.NH_FLAGS | (2 << 20), damping=0.005), pbd=dict(PBD),
              both=dict(PBD, flags=W.YEOH_FLAGS | (3 << 20), damping=0.005), volume=dict(volume_passes=2))


def _settings(flags=W.NH_FLAGS, **kw):
    return xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=W.nh_compliance(1e5, 0.45),
                                 poissons_ratio=0.45, flags=flags, **kw)


def _tets(*dims, pattern=0):
    nodes, idx = xfem.generate_tet_block(*dims, (0.05, 0.05, 0.05), pattern, 0.2)
    return nodes, idx, 1000.0


def _automatic(meshes, **opts):
    """A handle that times its forms and has not picked the colour graph (on a busy
    GPU that one can win)."""
    for _ in range(8):
        b = xfem.Body(meshes=meshes, settings=[_settings()] * len(meshes), **opts)
        b.step_frames(1, 20, DT)
        if b.info()["sync_mode"] != 2:
            return b
    pytest.skip("the GPU is busy: the colour graph was timed fastest eight times")


# One cluster: 16 blocks at most, a warp per chunk of a colour, two chunk buffers of
# 13.3 KB a warp and 32 bytes per vertex in 227 KB of shared memory. At 256 threads
# that is six warps a block: 96 chunks of a colour (64 x 24 x 16 cubes: 161 KB of
# buffers, 55 of vertices) do, 99 (seven warps: 188 and 57) and 128 do not.
@pytest.mark.parametrize("dims,block,form", [((1, 1, 1), 64, "cluster"), ((8, 2, 2), 128, "cluster"),
                                             ((17, 12, 11), 128, "cluster"), ((32, 16, 16), 64, "cluster"),
                                             ((64, 24, 16), 256, "cluster"), ((66, 24, 16), 256, "grid"),
                                             ((64, 32, 16), 256, "grid")])
@pytest.mark.parametrize("sweeps", ["plain", "both", "volume"])
def test_small_handles(dims, block, form, sweeps):
    s = _settings(**SWEEPS.get(sweeps, {}))
    a = xfem.Body(*_tets(*dims), s, sync_mode=1, block_size=block)
    assert a.launch()["form"] == "none"
    b = xfem.Body(*_tets(*dims), s, sync_mode=1, block_size=block, keep_lambdas=True)
    for h in (a, b):
        h.step_frames(1, 9, DT)
    got = a.launch()
    assert got["form"] == form and got["threads"] == block
    assert (got["blocks"] <= 16) == (form == "cluster")
    assert b.launch()["form"] == "grid"
    assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities(), b.velocities())
    a.step_frames_noalloc(1, 2, DT)
    assert a.launch()["form"] == "grid" and a.launch()["blocks"] == a.info()["blocks"]


@pytest.mark.parametrize("mesh", ["one_tet", "mirrored", "batch"])
def test_small_handles_of_other_chunks(mesh):
    meshes = [_tets(n, 6, 5, pattern=int(mesh == "mirrored")) for n in ((2, 5, 9) if mesh == "batch" else (7,))]
    b = xfem.Body(meshes=meshes, settings=[_settings()] * len(meshes), sync_mode=1, block_size=128,
                  cluster_mode=1 if mesh == "one_tet" else 0)
    b.step_frames(1, 2, DT)
    assert b.launch()["form"] == "cluster"


@pytest.mark.parametrize("mode,form", [(2, "graph"), (3, "dataflow"), (4, "bricks")])
def test_fixed_forms(mode, form):
    b = xfem.Body(*_tets(24, 16, 8), _settings(), sync_mode=mode, block_size=128)
    for n in (3, 3):
        b.step_frames(1, n, DT)
        assert b.launch()["form"] == form and b.launch()["blocks"] > 1


# the reverse as one cluster: up to two chunks of a colour per block (32 x 16 x 16: 32 in 16)
@pytest.mark.parametrize("dims,record,reverse,lanes", [
    ((8, 2, 2), "cluster", "cluster", 1), ((20, 9, 9), "cluster", "cluster", 1), ((32, 16, 12), "cluster", "cluster", 1),
    ((32, 16, 16), "cluster", "cluster", 1), ((32, 17, 16), "cluster", "grid", 8), ((32, 21, 20), "cluster", "grid", 8)])
def test_adjoint(dims, record, reverse, lanes, monkeypatch):
    b = xfem.Body(*_tets(*dims), _settings(), block_size=256)
    b.adjoint_forward(4, DT, np.uint32([0]))
    assert b.launch(xfem.LAUNCH_RECORD)["form"] == record
    g = np.ones((4, 1, 3), np.float32)
    b.adjoint_backward(g)
    got = b.launch(xfem.LAUNCH_REVERSE)
    assert got["form"] == reverse and got["lanes"] == lanes
    monkeypatch.setenv("XFEM_REVERSE_FORM", "lane")
    b.adjoint_backward(g)
    got = b.launch(xfem.LAUNCH_REVERSE)
    assert got["form"] == "grid" and got["lanes"] == 1


# meshes of tests/test_gpu_bricks_ext.py
@pytest.mark.parametrize("dims,block", [((49, 33, 31), 128), ((49, 33, 31), 256), ((96, 64, 40), 192)])
def test_sweeps_on_bricks(dims, block):
    b = _automatic([_tets(*dims)], block_size=block)
    for sweeps in sorted(SWEEPS):
        b.set_settings(_settings(**SWEEPS[sweeps]))
        b.step_frames(1, 2, DT)
        got = b.launch()
        assert got["form"] == "bricks_ext" and got["blocks"] == b.info()["bricks"] and got["threads"] == block, sweeps
    a = xfem.Body(*_tets(*dims), _settings(**DAMPED), sync_mode=1, block_size=256)
    a.step_frames(1, 2, DT)
    assert a.launch()["form"] == "grid"


def test_sweeps_on_bricks_wait_times_out_and_recovers():
    """A neighbour wait that expects one pass more than the bricks publish runs out
    after the short limit, and the handle steps normally afterwards."""
    mesh = _tets(49, 33, 31)
    b = _automatic([mesh], block_size=256, wait_timeout_ms=100)
    ref = xfem.Body(*mesh, _settings(), sync_mode=1, block_size=256)
    x0 = mesh[0].reshape(-1, 3)
    for h in (ref, b):  # the locks take hold in the first substep
        h.set_settings(_settings(**DAMPED))
        h.step_frames(1, 1, DT)
        h.set_positions(x0)
        h.set_velocities(np.zeros_like(x0))
    assert b.launch()["form"] == "bricks_ext"
    ref.step_frames(1, 6, DT)
    xfem.test_hook(b, xfem.HOOK_MISSING_ARRIVAL, 1)
    b.step_frames(1, 6, DT)
    with pytest.raises(xfem.XfemError) as e:
        b.synchronize()
    assert e.value.code == xfem.EDEVICE_TIMEOUT
    b.set_positions(x0)
    b.set_velocities(np.zeros_like(x0))
    b.step_frames(1, 6, DT)
    assert b.launch()["form"] == "bricks_ext"
    assert np.array_equal(b.positions(), ref.positions()) and np.array_equal(b.velocities(), ref.velocities())


def test_elements_and_rings():
    nodes, idx = xfem.generate_hex_block(4, 3, 3, (0.05, 0.05, 0.05), 0, 0.2)
    ring = 9 << xfem.ENERGY_BIT
    for flags, mesh, form, lanes in ((W.NH_FLAGS, (nodes, idx, 1000.0), "elements", 1),
                                     (W.NH_FLAGS | xfem.ELEMENT_H27, (nodes, idx, 1000.0), "elements", 32),
                                     (W.NH_FLAGS | xfem.ELEMENT_T10, _tets(4, 3, 3), "elements", 4),
                                     (ring, _tets(4, 3, 3), "rings", 32), (ring, (nodes, idx, 1000.0), "rings", 32),
                                     (ring | xfem.ELEMENT_T10, _tets(4, 3, 3), "rings", 32),
                                     (ring | xfem.ELEMENT_H27, (nodes, idx, 1000.0), "rings", 32)):
        b = xfem.Body(*mesh, _settings(flags=flags))
        b.step_frames(1, 2, DT)
        assert b.launch()["form"] == form and b.launch()["lanes"] == lanes, flags
        assert b.launch()["blocks"] >= 1


def _quadratic_kinds(flags, volume_passes):
    """Settings of every energy, coupled and serial, with every damping type."""
    out = []
    for k, energy in enumerate(2 * (4, 0, 7, 3, 1, 6, 2, 5, 11, 4, 7, 3, 0, 31, 12, 5)):
        out.append(xfem.default_settings(
            gravity=(0.3, -9.81, -2.0), compliance=4e-5 * (1 + k % 5), poissons_ratio=0.45,
            damping=0.0 if k % 3 == 0 else 0.002, pbd_damping=0.02 * (k % 2),
            volume_and_time_corrected_pbd_damping=0.01, amortized_volume_and_time_corrected_pbd_damping=0.05,
            volume_passes=volume_passes * (k % 2),
            flags=flags | (energy << xfem.ENERGY_BIT) | (((k + k // 4) % 4) << 20) | xfem.LOCK_LEFT |
            ((k % 5 != 1) << xfem.XPBD_SOLVE_BIT)))
    return out


def _coupled(flags):
    return _settings(flags=flags | W.NH_FLAGS)


@pytest.mark.parametrize("volume_passes", [0, 2])
def test_one_and_four_lane_t10s_of_every_energy(volume_passes):
    """Which kernel a handle of T10s takes follows from its largest colour and from what
    most of its T10s solve: bodies of every kind step alike in a batch that takes one lane
    per T10, in one that takes four, and alone."""
    kinds = _quadratic_kinds(xfem.ELEMENT_T10, volume_passes)
    mesh = xfem.generate_tet_block(12, 10, 9, (0.1, 0.1, 0.1), 0, 0.2) + (1000.0,)
    small = xfem.generate_tet_block(3, 2, 2, (0.1, 0.1, 0.1), 0, 0.2) + (1000.0,)
    one = xfem.Body(meshes=[mesh] * 48, settings=kinds + kinds[:16])
    # a few larger coupled bodies are most of the T10s
    four = xfem.Body(meshes=[small] * len(kinds) + [mesh], settings=kinds + [_coupled(xfem.ELEMENT_T10)])
    alone = [xfem.Body(*small, s) for s in kinds]
    for h in [one, four] + alone:
        h.step_frames(1, 9, DT)
    assert one.launch()["lanes"] == 1 and four.launch()["lanes"] == 4
    assert {a.launch()["lanes"] for a in alone} == {1, 4}
    for k, a in enumerate(alone):
        assert np.array_equal(a.positions(), four.positions(k)), k
        assert np.array_equal(a.velocities(), four.velocities(k)), k
    for k in (0, 1, 2, 3, 5, 6, 7, 9, 13, 17, 18, 22):  # and at the larger size
        lanes = xfem.Body(meshes=[mesh] * 3, settings=[kinds[k]] + 2 * [_coupled(xfem.ELEMENT_T10)])
        lanes.step_frames(1, 9, DT)
        assert lanes.launch()["lanes"] == 4
        assert np.array_equal(one.positions(k), lanes.positions(0)), k
        assert np.array_equal(one.velocities(k), lanes.velocities(0)), k
        assert np.isfinite(one.positions(k)).all(), k


@pytest.mark.parametrize("kw,lanes", [
    (dict(), 4), (dict(flags=W.YEOH_FLAGS), 4), (dict(damping=0.002), 1), (dict(pbd_damping=0.02), 4),
    (dict(damping=0.002, flags=W.NH_FLAGS | (2 << 20)), 4), (dict(volume_passes=2), 4),
    (dict(flags=(xfem.ENERGY_MIXED_SEL << xfem.ENERGY_BIT) | xfem.LOCK_LEFT), 1),
    (dict(flags=(xfem.ENERGY_MIXED << xfem.ENERGY_BIT) | xfem.LOCK_LEFT), 4),
    (dict(flags=(xfem.ENERGY_PIXAR << xfem.ENERGY_BIT) | xfem.LOCK_LEFT, damping=0.002), 4),
    (dict(flags=(xfem.ENERGY_PIXAR_SEL << xfem.ENERGY_BIT) | xfem.LOCK_LEFT, damping=0.002), 1)])
def test_lanes_per_t10_by_settings(kw, lanes):
    flags = kw.get("flags", W.NH_FLAGS) | xfem.ELEMENT_T10
    b = xfem.Body(*_tets(4, 3, 2), _settings(**{**kw, "flags": flags}))
    b.step_frames(1, 1, DT)
    assert b.launch()["lanes"] == lanes
    b.set_settings(_settings(flags=W.NH_FLAGS | xfem.ELEMENT_T10))
    b.step_frames(1, 1, DT)
    assert b.launch()["lanes"] == 4


def _tets_and_hexes(w, h, d, every):
    """A block of hexes, all but each `every`-th cell split into six tets."""
    nodes, idx = xfem.generate_hex_block(w, h, d, (0.1, 0.1, 0.1), 0, 0.2)
    six = ((0, 1, 5, 7), (0, 7, 3, 1), (0, 2, 3, 7), (0, 7, 6, 2), (0, 4, 6, 7), (0, 7, 5, 4))
    out = []
    for k, c in enumerate(idx.reshape(-1, 9)):
        if k % every == 0:
            out.extend(c)
        else:
            for t in six:
                out.append(4)
                out.extend(c[1:][list(t)])
    return nodes, np.array(out, np.uint32), 1000.0


@pytest.mark.parametrize("volume_passes", [0, 2])
def test_one_and_four_lane_t10s_beside_h27s(volume_passes):
    """The same on meshes mixing T10s and H27s."""
    kinds = _quadratic_kinds(xfem.ELEMENT_H27, volume_passes)
    mesh, small = _tets_and_hexes(12, 10, 9, 20), _tets_and_hexes(3, 3, 2, 4)
    one = xfem.Body(meshes=[mesh] * 40, settings=kinds + kinds[:8])
    four = xfem.Body(meshes=[small] * len(kinds) + [mesh], settings=kinds + [_coupled(xfem.ELEMENT_H27)])
    alone = [xfem.Body(*small, s) for s in kinds]
    for h in [one, four] + alone:
        h.step_frames(1, 9, DT)
    assert one.launch()["lanes"] == 1 and four.launch()["lanes"] == 4
    assert {a.launch()["lanes"] for a in alone} == {1, 4}
    for k, a in enumerate(alone):
        assert np.array_equal(a.positions(), four.positions(k)), k
        assert np.array_equal(a.velocities(), four.velocities(k)), k
    for k in (0, 1, 3, 5, 9, 13, 18):
        lanes = xfem.Body(meshes=[mesh] * 3, settings=[kinds[k]] + 2 * [_coupled(xfem.ELEMENT_H27)])
        lanes.step_frames(1, 9, DT)
        assert lanes.launch()["lanes"] == 4
        assert np.array_equal(one.positions(k), lanes.positions(0)), k
        assert np.array_equal(one.velocities(k), lanes.velocities(0)), k
        assert np.isfinite(one.positions(k)).all(), k


# most of the cells tets: up to one round of four-lane warps (8 T10s x 8 warps a SM), beyond it
@pytest.mark.parametrize("bodies,lanes", [(6, 4), (40, 1)])
def test_lanes_per_t10_beside_h27s_by_size(bodies, lanes):
    b = xfem.Body(meshes=[_tets_and_hexes(12, 10, 9, 20)] * bodies, settings=[_coupled(xfem.ELEMENT_H27)] * bodies)
    b.step_frames(1, 1, DT)
    assert b.launch()["lanes"] == lanes


def test_h27_rings_fill_the_sms():
    """A ring is one warp's chain, so large meshes need many warps in flight: 15 per SM,
    12 with damping (blocks of four with their own copy of the tables left 8)."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nodes, idx = xfem.generate_hex_block(5, 4, 3, (0.05, 0.05, 0.05), 0, 0.2)
    for kw in ({}, dict(damping=0.005), DAMPED):
        flags = (9 << xfem.ENERGY_BIT) | xfem.ELEMENT_H27 | (kw.get("flags", 0) & (3 << 20))
        b = xfem.Body(nodes, idx, 1000.0, _settings(**{**kw, "flags": flags}))
        b.step_frames(1, 2, DT)
        assert b.launch()["blocks"] * b.launch()["threads"] // 32 == (12 if kw else 15) * sms


@pytest.mark.parametrize("energy", [xfem.ENERGY_CUBE_NEO, xfem.ENERGY_CUBE_SKIN])
@pytest.mark.parametrize("opts", [dict(sync_mode=1, block_size=128), dict(sync_mode=2, block_size=128),
                                  dict(sync_mode=1, block_size=128, keep_lambdas=True),
                                  dict(sync_mode=2, block_size=128, cluster_mode=1, keep_lambdas=True)])
def test_cube_models_leave_tets_alone(energy, opts):
    """Every vertex of a tet mesh with a cube model falls as one, and the multipliers
    are zero, in the forms of whole cubes and of single tets."""
    nodes, idx, density = _tets(9, 7, 5)
    s = _settings(flags=(energy << xfem.ENERGY_BIT) | (1 << xfem.XPBD_SOLVE_BIT))
    b = xfem.Body(nodes, idx, density, s, **opts)
    b.step_frames(1, 6, DT)
    assert b.launch()["form"] == ("graph" if opts["sync_mode"] == 2 else "grid" if "keep_lambdas" in opts else "cluster")
    v = b.velocities()
    # each substep rounds (v + g dt) drag and the position it is taken from: a few ulps of x / dt
    tol = 6 * 4 * 2.0 ** -24 * np.abs(nodes).max() / DT
    assert np.abs(v - v.mean(0)).max() <= tol and v[:, 1].max() < -6 * 9.0 * DT
    if "keep_lambdas" in opts:
        assert not b.lambdas().any()


def test_a_handle_follows_its_settings_off_the_bricks_and_back():
    """A damped handle whose sweeps run on the bricks keeps them when the damping is
    switched off, takes a form with the extended solves for the Pixar models, and comes
    back; each time it steps as a handle that stays on the grid."""
    mesh = _tets(49, 33, 31)
    b = None
    for _ in range(8):  # its forms are timed: on a busy GPU another one can win
        b = xfem.Body(*mesh, _settings(**DAMPED))
        b.step_frames(1, 20, DT)
        if b.launch()["form"] == "bricks_ext":
            break
    else:
        pytest.skip("the GPU is busy: another form was timed fastest eight times")
    a = xfem.Body(*mesh, _settings(**DAMPED), sync_mode=1, block_size=256)
    a.step_frames(1, 20, DT)
    pixar = _settings(flags=(xfem.ENERGY_PIXAR_SEL << xfem.ENERGY_BIT) | (1 << xfem.XPBD_SOLVE_BIT) | xfem.LOCK_LEFT)
    plain, damped = _settings(), _settings(**DAMPED)
    for s, forms in ((plain, ["bricks"]), (damped, ["bricks_ext"]), (pixar, ["graph", "grid"]), (plain, ["bricks"]),
                     (pixar, ["graph", "grid"]), (damped, ["bricks_ext"]), (pixar, ["graph", "grid"]),
                     (damped, ["bricks_ext"]), (plain, ["bricks"])):
        for h in (a, b):
            h.set_settings(s)
            h.step_frames(1, 3, DT)
        assert b.launch()["form"] in forms
        assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities(), b.velocities())


def test_brick_tables_of_the_sweeps_are_built_when_needed():
    """A handle that never damps does not hold the sweeps' tables on the bricks; one that
    cannot allocate them sweeps on the grid, and on the bricks once it can."""
    mesh = _tets(49, 33, 31)
    b = _automatic([mesh], block_size=256)
    a = xfem.Body(*mesh, _settings(), sync_mode=1, block_size=256)
    a.step_frames(1, 20, DT)
    plain, damped = _settings(), _settings(**DAMPED)
    before = b.info()["device_bytes"]
    for s, fail, form in ((damped, True, "grid"), (plain, False, None), (damped, False, "bricks_ext"), (plain, False, "bricks")):
        if fail:
            xfem.test_hook(None, xfem.HOOK_FAIL_ALLOC, 1)
        for h in (b, a):
            h.set_settings(s)
            h.step_frames(1, 3, DT)
        if form:
            assert b.launch()["form"] == form
        assert (b.info()["device_bytes"] > before) == (form in ("bricks_ext", "bricks"))
        assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities(), b.velocities())


def test_a_handle_tuned_with_a_pixar_model_steps_plain_bodies_on_the_bricks():
    mesh = _tets(49, 33, 31)
    pixar = _settings(flags=(xfem.ENERGY_PIXAR_SEL << xfem.ENERGY_BIT) | (1 << xfem.XPBD_SOLVE_BIT) | xfem.LOCK_LEFT)
    a = xfem.Body(*mesh, pixar, sync_mode=1, block_size=256)
    b = xfem.Body(*mesh, pixar)
    forms = []
    for s in (pixar, _settings(), pixar, _settings(**DAMPED), _settings(), pixar):
        for h in (a, b):
            h.set_settings(s)
            h.step_frames(1, 3, DT)
        forms.append(b.launch()["form"])
        assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities(), b.velocities())
    assert forms[1] == forms[4] == "bricks" and forms[3] == "bricks_ext"
    assert {forms[0], forms[2], forms[5]} <= {"graph", "grid"} and forms[0] == forms[2] == forms[5]


def test_a_handle_tuned_plain_returns_to_its_form():
    mesh = _tets(49, 33, 31)
    b = xfem.Body(*mesh, _settings())
    b.step_frames(1, 20, DT)
    first = b.launch()
    for s in (_settings(**DAMPED), _settings(), _settings(flags=W.NH_FLAGS | xfem.LOCK_RIGHT)):
        b.set_settings(s)
        b.step_frames(1, 3, DT)
    assert b.launch() == first


# one brick per SM of few chunks with slots for every vertex of its own (generic accesses); a
# chosen number of bricks: with more chunks, and with vertices that get no slot (the branch)
@pytest.mark.parametrize("bodies", [1, 2])
@pytest.mark.parametrize("dims,bricks", [((40, 24, 20), 0), ((40, 24, 20), 9), ((48, 32, 24), 3)])
def test_chosen_numbers_of_bricks(dims, bricks, bodies):
    meshes = [_tets(*dims)] * bodies
    s = [_settings(ground=1, ground_normal=(0.0, 1.0, 0.0), ground_offset=-0.01, friction=0.4)] * bodies
    a = xfem.Body(meshes=meshes, settings=s, sync_mode=1, block_size=256)
    b = xfem.Body(meshes=meshes, settings=s, sync_mode=4, block_size=256, bricks=bricks)
    for n in (7, 2):
        for h in (a, b):
            h.step_frames(1, n, DT)
    assert b.launch()["form"] == "bricks" and (not bricks or b.launch()["blocks"] == bricks)
    for k in range(bodies):
        assert np.array_equal(a.positions(k), b.positions(k)) and np.array_equal(a.velocities(k), b.velocities(k))


def test_a_chosen_number_of_bricks_is_for_sync_mode_4():
    """The sweeps of an automatic handle stay off bricks whose number the caller chose."""
    b = xfem.Body(*_tets(49, 33, 31), _settings(), bricks=3)
    b.step_frames(1, 5, DT)
    b.set_settings(_settings(**DAMPED))
    b.step_frames(1, 2, DT)
    assert b.launch()["form"] in ("grid", "graph")
