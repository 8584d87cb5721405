"""GPU quadratic-tet mode: T10s (xfem_t10.cu) through the C ABI.

A tet mesh with element type T10 in flags bits 0-3 runs as GeoQuadratic3d
(XPBDFEM/Geo.cpp:836-1053): one node on every edge, SolveElement on
ElementParamsQuadraticTet with Nodes = 10 and the 4-point rule
(XPBDFEM/Fem.cpp:871-893), the Pixar models, Mixed, MixedSel and the Yeoh
models, coupled or serial, in-solve and post-step damping, PBD damping and
volume passes; the cube models leave a T10 alone.

Against the reference's own substeps run in the GPU body's T10 colour order
(the `qordered_*` and `qdamped_*` fixtures) and against the pinned oracle on
larger jittered blocks. Compressible materials: positions within 1e-5 of max
|x_ref| and velocities 1e-3 relative. With an incompressible material or
volume passes the FP32 rounding of J decides the result already within the
first substep on T10s (the reference's own FP32 run is 2.3e-3 from the FP64
run after one substep of the incompressible fixture, and FP32 runs from
1-ulp perturbed starts spread over 3e-3 to 5e-3), so those are checked
against the FP64 run of the same method and order: within 3x the spread of
FP32 runs (the reference's own run and perturbed starts) after one substep
and after all of them. Launch forms, call splits and batching agree bit for
bit.
"""
import numpy as np
import pytest

import oracle
import xfem
from conftest import golden, golden_args
from helpers import T10OracleRun, envelope, rel

pytestmark = pytest.mark.gpu

DT = 1.0 / 1200.0
QFIX = ["qordered_c1_nh_nu045", "qordered_c1_nh_incompressible", "qordered_wonky_yeohfast_serial_nu049",
        "qordered_c1_mixed_nu045", "qdamped_c1_nh_nu045_amortized_pbd", "qdamped_c1_pixar_nu045_limit",
        "qvolume_wonky_nh_serial_1_post"]


def copy_settings(s):
    return xfem.default_settings(**{k: getattr(s, k) for k, _ in s._fields_})


def t10_settings(name):
    """Settings of a `qordered` / `qdamped` fixture (refgen's argument order),
    with the element type T10."""
    a = golden_args(name)["args"]
    g = golden(name)
    dens, energy, simul, comp, nu, gx, gy, dt, nsub, lock = a[9:19]
    kw = dict(rtype=2, damping=0.0, pbd=0.0, drag=0.0, vc=0.0, avc=0.0, vp=0)
    if a[0] == "qdamped":
        d = g["derived"]
        kw = dict(damping=a[19], pbd=a[20], rtype=a[22], drag=float(d[2]), vc=float(d[0]), avc=float(d[1]),
                  vp=a[24] if len(a) > 24 else 0)
    flags = (xfem.ELEMENT_T10 | (energy << xfem.ENERGY_BIT) | (simul << xfem.XPBD_SOLVE_BIT) |
             (xfem.LOCK_LEFT if lock else 0) | (kw["rtype"] << 20))
    s = xfem.default_settings(gravity=(gx, gy, 0.0), compliance=comp, poissons_ratio=nu, flags=flags,
                              damping=kw["damping"], pbd_damping=kw["pbd"], time_corrected_drag=kw["drag"],
                              volume_and_time_corrected_pbd_damping=kw["vc"],
                              amortized_volume_and_time_corrected_pbd_damping=kw["avc"], volume_passes=kw["vp"])
    return g, s, dens, dt, nsub


@pytest.mark.parametrize("name", QFIX)
def test_t10_reference_parity(name):
    g, s, dens, dt, nsub = t10_settings(name)
    b = xfem.Body(g["nodes"], g["idx"], dens, s)
    nt, ne = b.t10_count()
    assert nt == g["order"].size and b.counts[0][0] == g["x1"].size // 3
    sch = b.t10_schedule()
    assert np.array_equal(sch["t10_order"], g["order"])
    assert np.array_equal(sch["colour_t10_begin"], g["colour_tet_begin"])
    b.substep(dt)
    x1, v1 = b.positions(), b.velocities()
    b.step_frames(1, nsub - 1, dt)
    xn, vn = b.positions(), b.velocities()
    if s.poissons_ratio >= 0.5 or s.volume_passes:
        # within 3x the FP32 spread (the reference's own run included) about
        # the FP64 run of the same method and order, after one substep and
        # after all of them
        ref, env = envelope(lambda dt_: T10OracleRun(g["nodes"], g["idx"], dens, copy_settings(s), g["order"],
                                                     dtype=dt_), (1, nsub), dt)
        (X1_64, V1_64), (Xn_64, _) = ref
        ex1 = max(env[0][0], rel(g["x1"].reshape(-1, 3), X1_64))
        ev1 = max(env[0][1], rel(g["v1"].reshape(-1, 3), V1_64))
        exn = max(env[1][0], rel(g["xn"].reshape(-1, 3), Xn_64))
        assert rel(x1, X1_64) <= 3 * ex1 + 1e-7
        assert rel(v1, V1_64) <= 3 * ev1 + 1e-7
        assert rel(xn, Xn_64) <= 3 * exn + 1e-7
        return
    assert rel(x1, g["x1"].reshape(-1, 3)) <= 1e-5
    assert rel(v1, g["v1"].reshape(-1, 3)) <= 1e-3
    assert rel(xn, g["xn"].reshape(-1, 3)) <= 1e-5
    assert rel(vn, g["vn"].reshape(-1, 3)) <= 1e-3


@pytest.mark.parametrize("energy,simultaneous,comp,nu,vpasses,damping,rtype,pbd", [
    (xfem.ENERGY_MIXED_SEL, 1, 1e-3, 0.45, 0, 0.0, 2, 0.0),
    (xfem.ENERGY_MIXED_SEL, 0, 1e-3, 0.40, 0, 0.01, 0, 0.0),
    (xfem.ENERGY_YEOH_SKIN_FAST, 1, 0.5, 0.45, 0, 0.01, 1, 0.0),
    (xfem.ENERGY_MIXED, 1, 1e-3, 0.45, 0, 0.01, 3, 0.03),
    (xfem.ENERGY_YEOH_SKIN, 0, 0.5, 0.45, 0, 0.01, 2, 0.0),
    (xfem.ENERGY_YEOH_SKIN_SEL, 1, 0.5, 0.49, 0, 0.0, 2, 0.05),
    (xfem.ENERGY_PIXAR, 1, 1e-3, 0.45, 0, 0.0, 2, 0.0),
    (xfem.ENERGY_PIXAR_SEL, 1, 1e-3, 0.40, 0, 0.01, 2, 0.0),
    (20, 1, 1e-3, 0.45, 0, 0.0, 2, 0.0),
    (xfem.ENERGY_CUBE_NEO, 1, 1e-3, 0.45, 0, 0.01, 3, 0.03),
    (xfem.ENERGY_MIXED_SEL, 1, 1e-3, 0.45, 1, 0.01, 2, 0.0),
])
def test_t10_oracle_parity(energy, simultaneous, comp, nu, vpasses, damping, rtype, pbd):
    """A larger jittered mirrored block, 20 substeps, against the oracle in
    the body's own T10 order."""
    nodes, idx = xfem.generate_tet_block(5, 3, 3, (0.05, 0.05, 0.05), 1, 0.2)
    rng = np.random.default_rng(5)
    nodes = (nodes + rng.normal(0, 0.002, nodes.shape)).astype(np.float32)
    flags = (xfem.ELEMENT_T10 | (energy << xfem.ENERGY_BIT) | (simultaneous << xfem.XPBD_SOLVE_BIT) |
             xfem.LOCK_LEFT | (rtype << 20))
    vc, avc = xfem.pbd_damping_coefficients(pbd, DT, 0.05)
    s = xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=comp, poissons_ratio=nu, flags=flags,
                              damping=damping, pbd_damping=pbd, volume_and_time_corrected_pbd_damping=vc,
                              amortized_volume_and_time_corrected_pbd_damping=avc, volume_passes=vpasses)
    b = xfem.Body(nodes, idx, 800.0, s)
    order = b.t10_schedule()["t10_order"]
    if vpasses:
        # volume passes: within 3x the FP32 spread about the FP64 run
        ref, env = envelope(lambda dt_: T10OracleRun(nodes, idx, 800.0, copy_settings(s), order, dtype=dt_),
                            (1, 20), DT)
        for k, n in enumerate((1, 19)):
            b.step_frames(1, n, DT)
            assert rel(b.positions(), ref[k][0]) <= 3 * env[k][0] + 1e-7, n
            assert rel(b.velocities(), ref[k][1]) <= 3 * env[k][1] + 1e-7, n
        return
    o = T10OracleRun(nodes, idx, 800.0, s, order)
    for n in (1, 19):
        b.step_frames(1, n, DT)
        o.step(n, DT)
        o.s.tick_id += n
        assert rel(b.positions(), o.X) <= 1e-5, n
        assert rel(b.velocities(), o.V) <= 1e-3, n


def test_t10_rest_state_and_volume():
    nodes, idx = xfem.generate_tet_block(4, 3, 2, (0.04, 0.05, 0.06), 1, 0.3)
    s = xfem.default_settings(flags=xfem.default_settings().flags | xfem.ELEMENT_T10)
    b = xfem.Body(nodes, idx, 900.0, s)
    ep, w, t10, edges = b.t10_rest_state()
    x, e2, w2, _ = xfem.compute_t10_rest_state(nodes, idx, 900.0)
    assert np.array_equal(ep.view(np.uint32), e2.view(np.uint32))
    assert np.array_equal(w.view(np.uint32), w2.view(np.uint32))
    assert np.array_equal(b.inverse_masses().view(np.uint32), w2.view(np.uint32))
    e3, t3 = xfem.compute_t10_edges(idx)
    assert np.array_equal(edges, e3) and np.array_equal(t10, t3)
    # the body's rest positions: the mesh's own, then the edge midpoints
    assert np.array_equal(b.positions(), x.astype(np.float32))
    q = oracle.Quadratic(nodes, idx, 900.0, np.float64)
    assert abs(b.volume() - q.volume(b.positions().astype(np.float64))) <= 1e-6 * b.volume()
    s.flags &= ~xfem.LOCK_LEFT
    s.gravity[1] = -9.81
    b.set_settings(s)
    b.step_frames(2, 10, DT)
    assert abs(b.volume() - q.volume(b.positions().astype(np.float64))) <= 1e-6 * b.volume()


def test_t10_launch_forms_agree():
    """One call, one call per substep, and the allocation-free launch."""
    g, s, dens, dt, nsub = t10_settings("qdamped_c1_nh_nu045_amortized_pbd")
    runs = []
    for form in ("frames", "split", "noalloc"):
        b = xfem.Body(g["nodes"], g["idx"], dens, s)
        if form == "frames":
            b.step_frames(1, nsub, dt)
        elif form == "split":
            for _ in range(nsub):
                b.substep(dt)
        else:
            b.step_frames_noalloc(1, nsub, dt)
        runs.append((b.positions(), b.velocities()))
    for x, v in runs[1:]:
        assert np.array_equal(x, runs[0][0])
        assert np.array_equal(v, runs[0][1])


def test_t10_batch_each_as_alone():
    """T10 bodies with different models, damping and volume passes in one
    handle: each as when run alone."""
    names = ["qvolume_wonky_nh_serial_1_post", "qdamped_c1_pixar_nu045_limit", "qordered_c1_mixed_nu045",
             "qordered_wonky_yeohfast_serial_nu049"]
    meshes, settings, alone = [], [], []
    for name in names:
        g, s, dens, dt, nsub = t10_settings(name)
        b = xfem.Body(g["nodes"], g["idx"], dens, s)
        b.step_frames(1, 12, DT)
        alone.append((b.positions(), b.velocities()))
        meshes.append((g["nodes"], g["idx"], dens))
        settings.append(s)
    B = xfem.Body(meshes=meshes, settings=settings)
    B.step_frames(1, 12, DT)
    for k in range(len(meshes)):
        assert np.array_equal(B.positions(k), alone[k][0]), k
        assert np.array_equal(B.velocities(k), alone[k][1]), k


def test_t10_errors():
    nodes, idx = xfem.generate_tet_block(3, 2, 2, (0.05, 0.05, 0.05))
    hn, hi = xfem.generate_hex_block(3, 2, 2, (0.05, 0.05, 0.05))
    t10 = xfem.default_settings().flags | xfem.ELEMENT_T10
    # the continuous-pressure models run on T10s (tests/test_gpu_t10_rings.py);
    # switching to them under an element-model handle needs a new handle
    ring = xfem.Body(nodes, idx, 1000.0, xfem.default_settings(flags=xfem.ELEMENT_T10 | (9 << xfem.ENERGY_BIT)))
    assert ring.ring_schedule()["vert_order"].size == nodes.size // 3
    elem = xfem.Body(nodes, idx, 1000.0, xfem.default_settings(flags=t10))
    with pytest.raises(xfem.XfemError) as ex:
        elem.set_settings(xfem.default_settings(flags=xfem.ELEMENT_T10 | (9 << xfem.ENERGY_BIT)))
    assert ex.value.code == xfem.EUNSUPPORTED
    # element type T10 on a hex mesh makes quadratic hexes, as in the reference
    assert xfem.Body(hn, hi, 1000.0, xfem.default_settings(flags=t10)).h27_count()[0] == 12
    # linear and quadratic tets cannot share a handle
    with pytest.raises(xfem.XfemError) as ex:
        xfem.Body(meshes=[(nodes, idx, 1000.0), (nodes, idx, 1000.0)],
                  settings=[xfem.default_settings(flags=t10), xfem.default_settings()])
    assert ex.value.code == xfem.EUNSUPPORTED
    b = xfem.Body(nodes, idx, 1000.0, xfem.default_settings(flags=t10))
    # the element type cannot change under a handle
    with pytest.raises(xfem.XfemError) as ex:
        b.set_settings(xfem.default_settings())
    assert ex.value.code == xfem.EUNSUPPORTED
    for call in (lambda: b.set_tet_mu(np.ones(60, np.float32)), lambda: b.rest_state(), lambda: b.schedule(),
                 lambda: b.hex_rest_state(), lambda: b.adjoint_forward(2, DT, np.array([0], np.uint32))):
        with pytest.raises(xfem.XfemError) as ex:
            call()
        assert ex.value.code == xfem.EUNSUPPORTED
    b.step_frames(1, 4, DT)
    assert np.isfinite(b.positions()).all()


@pytest.mark.parametrize("volume_passes", [0, 2])
def test_bodies_of_every_energy_share_a_warp(volume_passes):
    """Eight T10s of a colour share a warp, four lanes each, whatever their
    bodies' energies: small bodies of every energy, coupled and serial, damped
    in the solve, after it and not at all, in one handle step as alone."""
    meshes, settings = [], []
    for k, energy in enumerate((4, 0, 7, 3, 1, 6, 2, 5, 11, 4, 7, 3, 0, 31)):
        dims = ((1, 1, 1), (2, 1, 1), (3, 2, 1))[k % 3]
        nodes, idx = xfem.generate_tet_block(*dims, (0.1, 0.1, 0.1), k % 2, 0.2)
        rtype = k % 4
        s = xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=4e-5 * (1 + k), poissons_ratio=0.45,
                                  damping=0.0 if k % 3 == 0 else 0.003, pbd_damping=0.02 * (k % 2),
                                  volume_and_time_corrected_pbd_damping=0.01,
                                  amortized_volume_and_time_corrected_pbd_damping=0.05, volume_passes=volume_passes * (k % 2),
                                  flags=xfem.ELEMENT_T10 | (energy << xfem.ENERGY_BIT) | (rtype << 20) | xfem.LOCK_LEFT |
                                  ((k % 5 != 1) << xfem.XPBD_SOLVE_BIT))
        meshes.append((nodes, idx, 1000.0))
        settings.append(s)
    batch = xfem.Body(meshes=meshes, settings=settings)
    batch.step_frames(1, 11, DT)
    for k, (m, s) in enumerate(zip(meshes, settings)):
        one = xfem.Body(*m, s)
        one.step_frames(1, 11, DT)
        assert np.array_equal(one.positions(), batch.positions(k)), k
        assert np.array_equal(one.velocities(), batch.velocities(k)), k
        assert np.isfinite(one.positions()).all()


def test_a_colour_beyond_one_round_steps_like_a_small_one():
    """Meshes whose largest colour needs a second round of four-lane warps take
    a lane per T10 (xfem_t10_lane.cu): a batch large enough for that steps its
    bodies as each alone (four lanes) does."""
    meshes, settings = [], []
    for k in range(48):
        nodes, idx = xfem.generate_tet_block(12, 10, 9, (0.1, 0.1, 0.1), 0, 0.2)
        s = xfem.default_settings(gravity=(0.3, -9.81, -2.0), compliance=4e-5 * (1 + k % 3), poissons_ratio=0.45,
                                  damping=0.002 * (k == 1), volume_passes=int(k == 2), pbd_damping=0.02 * (k == 3),
                                  volume_and_time_corrected_pbd_damping=0.01,
                                  flags=xfem.ELEMENT_T10 | ((4, 7, 3)[k % 3] << xfem.ENERGY_BIT) | (2 << 20) |
                                  xfem.LOCK_LEFT | ((k != 5) << xfem.XPBD_SOLVE_BIT))
        meshes.append((nodes, idx, 1000.0))
        settings.append(s)
    batch = xfem.Body(meshes=meshes, settings=settings)
    sched = np.diff(batch.t10_schedule()["colour_t10_begin"]).max() * len(meshes)
    assert sched > 8 * 12 * 160
    batch.step_frames(1, 3, DT)
    for k in range(6):
        one = xfem.Body(*meshes[k], settings[k])
        one.step_frames(1, 3, DT)
        assert np.array_equal(one.positions(), batch.positions(k)), k
        assert np.array_equal(one.velocities(), batch.velocities(k)), k
