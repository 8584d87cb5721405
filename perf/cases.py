"""The work that a user of xfem has it do, as cases to time and to compare.

Every case steps bodies through the public Python interface (xfem.Body): a
frame of substeps, then the positions and velocities read back into page-locked
arrays, as a simulation loop does; the gradient case runs the recording forward
and the reverse pass on a new set of inputs. Meshes are the generator's boxes
with jittered nodes (the repository's own workloads), or a box whose tets and
vertices come in random order, as from a mesher that knows no grid. All sizes
are cubes per side.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call, run() is one pass, work() what the pass
cannot do without, and exact() the same results in 64 bits, from the method
written out here in plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xpbd-fem_gb300"))
import xfem  # noqa: E402

FRAME = 1.0 / 60.0
DENSITY = 1000.0
TIPS = 20
YEOH = (1.0, 1.0 / 30.0, 1.0 / 300.0)  # C20 / C10 and C30 / C10 of the drop's 3e4, 1e3, 1e2 Pa
ENERGY = {"nh": xfem.ENERGY_MIXED_SEL, "yeoh": xfem.ENERGY_YEOH_SKIN_FAST, "mixed": xfem.ENERGY_MIXED,
          "ring": xfem.ENERGY_CONTINUOUS_MIXED}
# the six tets of a cube around its 0-7 diagonal; corners numbered i + 2j + 4k
SPLIT = np.array([[0, 1, 5, 7], [0, 7, 3, 1], [0, 2, 3, 7], [0, 7, 6, 2], [0, 4, 6, 7], [0, 7, 5, 4]])


def listed():
    def case(name, kind, w, h, d, **kw):
        c = dict(name=name, kind=kind, w=w, h=h, d=d, energy="nh", nu=0.45, substeps=20, young=1e5, edge=0.1)
        c.update(kw)
        return c

    return [
        # the smallest body (192 tets): a cantilever in an interactive scene, one frame at a time
        case("cantilever", "frame", 8, 2, 2, nu=0.5),
        # the reference's live loop: one call per substep, its web page's default damping
        case("interactive", "calls", 16, 8, 8, energy="yeoh", substeps=10, damping="ui"),
        # a body dropped onto a frictional ground (98,304 tets), 30 substeps a frame
        case("drop", "frame", 64, 16, 16, energy="yeoh", nu=0.5, substeps=30, young=1.8e5, edge=0.02, ground=True),
        # the headline mesh: 1,572,864 incompressible tets
        case("throughput", "frame", 128, 64, 32, nu=0.5, young=5e5),
        # a mesh with no grid in its numbering: clusters of every shape
        case("unstructured", "frame", 32, 24, 17, mesh="shuffled"),
        # the web page's default damping on a large body
        case("damped", "frame", 96, 33, 32, young=5e5, damping="ui"),
        # many bodies of uneven size in one handle, several frames between reads
        case("batched", "batch", 24, 24, 24, bodies=96, frames=4, edge=0.02, ground=True, young=2e4),
        # the gradient of a trajectory: 12,288 tets, 200 substeps, forward and reverse
        case("gradient", "adjoint", 32, 8, 8, substeps=200, edge=0.025),
        # linear hexahedra on the headline grid
        case("hexes", "frame", 128, 64, 32, element="hex", young=5e5),
        # quadratic tets (T10)
        case("t10", "frame", 48, 32, 25, element="t10"),
        # quadratic hexahedra (H27)
        case("h27", "frame", 48, 25, 24, element="h27"),
        # continuous-pressure model: one solve per vertex one-ring
        case("rings", "frame", 64, 32, 17, energy="ring", young=5e5),
    ]


def draw(rng):
    """One more case: the same kinds, sizes spread over their logarithm, ragged sides."""
    kind = rng.choice(["frame", "frame", "frame", "hex", "t10", "h27", "ring", "shuffled", "ui", "calls", "batch",
                       "adjoint"])
    # cubes of the smallest and the largest body of each kind
    lo, hi = {"frame": (32, 262144), "hex": (32, 262144), "t10": (32, 38400), "h27": (16, 28800), "ring": (32, 34816),
              "shuffled": (32, 13056), "ui": (64, 101376), "calls": (32, 4096), "batch": (64, 4096),
              "adjoint": (32, 8192)}[kind]
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    fx, fy = math.exp(rng.uniform(0.0, 1.0)), math.exp(rng.uniform(-0.4, 0.4))
    side = n ** (1.0 / 3.0)
    w = max(2, int(side * fx))
    h = max(1, int(side * fy / math.sqrt(fx)))
    d = max(1, int(n / (w * h)))
    edge, substeps = rng.choice([0.02, 0.05, 0.1]), rng.choice([5, 10, 15, 20])
    # a stiffness that the substep resolves: the wave speed times the substep stays below a fifth of an
    # edge (a tenth for quadratic elements, whose nodes are half as far apart)
    young = math.exp(rng.uniform(math.log(5e4), math.log(5e5))) * (edge / 0.1 * substeps / 20.0) ** 2
    c = dict(kind=kind if kind in ("calls", "batch", "adjoint") else "frame", w=w, h=h, d=d, energy="nh", nu=0.45,
             substeps=substeps, young=young * (0.2 if kind in ("t10", "h27") else 1.0), edge=edge)
    if kind == "frame":
        c.update(energy=rng.choice(["nh", "yeoh"]), ground=rng.random() < 0.4, nu=rng.choice([0.45, 0.45, 0.5]))
    elif kind in ("hex", "t10", "h27"):
        c.update(element=kind, energy=rng.choice(["nh", "nh", "yeoh", "mixed"] if kind == "hex" else ["nh", "yeoh"]))
    elif kind == "ring":
        c.update(energy="ring")
    elif kind == "shuffled":
        c.update(mesh="shuffled", energy=rng.choice(["nh", "yeoh"]))
    elif kind in ("ui", "calls"):
        c.update(damping="ui", energy=rng.choice(["nh", "yeoh"]))
    elif kind == "batch":
        side = max(3, int(side))
        c.update(w=side, h=side, d=side, bodies=rng.randint(2, 96), frames=rng.randint(1, 4), ground=True)
    elif kind == "adjoint":
        c.update(substeps=rng.randint(20, 200), edge=0.025, young=1e5)
    return c


# ---- meshes -------------------------------------------------------------------
def cubes(w, h, d):
    """Corner ids (i + 2j + 4k) of the cubes of a w x h x d grid, x fastest."""
    z, y, x = np.meshgrid(np.arange(d), np.arange(h), np.arange(w), indexing="ij")
    sx, sxy = w + 1, (w + 1) * (h + 1)
    base = (x + y * sx + z * sxy).reshape(-1, 1)
    return base + np.array([i + j * sx + k * sxy for k in (0, 1) for j in (0, 1) for i in (0, 1)])


def grid_nodes(w, h, d, edge, g):
    z, y, x = np.meshgrid(np.arange(d + 1), np.arange(h + 1), np.arange(w + 1), indexing="ij")
    p = edge * np.stack([x, y, z], -1).reshape(-1, 3)
    return p + (0.05 * edge) * g.standard_normal(p.shape)


def rotation(g):
    q, r = np.linalg.qr(g.standard_normal((3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else -q


def body_inputs(case, g, w, h, d):
    """(nodes[nv, 3] float32, elements, velocities[nv, 3] float32) of one body."""
    element, cs = case.get("element", "tet"), cubes(w, h, d)
    nodes = grid_nodes(w, h, d, case["edge"], g)
    el = cs if element in ("hex", "h27") else cs[:, SPLIT].reshape(-1, 4)
    if case.get("ground"):
        # turned at random, its lowest point just above the plane z = 0, falling
        nodes = (nodes - nodes.mean(0)) @ rotation(g).T
        nodes[:, 2] += 0.02 * case["edge"] - nodes[:, 2].min()
        v = np.tile(g.uniform(-0.2, 0.2, 3) - [0.0, 0.0, 1.0], (len(nodes), 1))
    else:
        # fixed at x = min, the rest swinging
        s = (nodes[:, :1] - nodes[:, 0].min()) / (nodes[:, 0].max() - nodes[:, 0].min())
        v = 0.3 * s * s * g.uniform(-1.0, 1.0, 3)
    if case.get("mesh") == "shuffled":
        new = g.permutation(len(nodes))  # vertex i becomes new[i]
        back = np.argsort(new)
        nodes, v, el = nodes[back], v[back], new[el][g.permutation(len(el))]
    return nodes.astype(np.float32), el, v.astype(np.float32)


def inputs(case, seed):
    """The bodies of a case (see body_inputs), its Young's moduli and, for the
    gradient, the per-tet moduli, the tip vertices and their target."""
    g = np.random.default_rng(seed)
    n = case.get("bodies", 1)
    if n == 1:
        bodies = [body_inputs(case, g, case["w"], case["h"], case["d"])]
        young = [case["young"]]
        energy = [case["energy"]]
    else:
        # the sizes are the case's, the rest the seed's
        dims = np.random.default_rng(n).integers(2, np.array([case["w"], case["h"], case["d"]]) + 1, (n, 3))
        bodies = [body_inputs(case, g, *(int(v) for v in x)) for x in dims]
        young = np.exp(g.uniform(math.log(0.1), math.log(10.0), n) + math.log(case["young"])).tolist()
        energy = ["yeoh" if x < 0.5 else "nh" for x in g.random(n)]
    out = dict(bodies=bodies, young=young, energy=energy)
    if case["kind"] == "adjoint":
        x = bodies[0][0]
        nt = len(bodies[0][1])
        mu = np.exp(math.log(case["young"]) + 0.3 * g.standard_normal(nt)) / (4.0 * (1.0 + case["nu"]))
        face = np.argsort(-x[:, 0], kind="stable")[:(case["h"] + 1) * (case["d"] + 1)]
        tips = face[np.linspace(0, len(face) - 1, min(TIPS, len(face))).round().astype(np.int64)]
        target = x[tips] + 0.5 * case["edge"] * g.standard_normal(3)
        out.update(mu=mu.astype(np.float32), tips=tips.astype(np.uint32), target=target.astype(np.float32))
    return out


def damping_of(case):
    """The reference's web page defaults (damping 0.005, PBD damping 0.03, drag 0.002)."""
    if case.get("damping") != "ui":
        return {}
    dt = FRAME / case["substeps"]
    pbd, amortized = xfem.pbd_damping_coefficients(0.03, dt, case["edge"])
    return dict(damping=0.005, pbd_damping=0.03, time_corrected_drag=xfem.time_corrected_drag(0.002, dt),
                volume_and_time_corrected_pbd_damping=pbd, amortized_volume_and_time_corrected_pbd_damping=amortized)


def compliance(case, young):
    return 4.0 * (1.0 + case["nu"]) / young  # mu = E / (4 (1 + nu)), the reference's scalar


def settings_of(case, young, energy):
    flags = (ENERGY[energy] << xfem.ENERGY_BIT) | (1 << xfem.XPBD_SOLVE_BIT)
    if not case.get("ground"):
        flags |= xfem.LOCK_LEFT
    if case.get("damping") == "ui":
        flags |= 3 << 20  # element damping of one eighth of the order per substep
    flags |= {"t10": xfem.ELEMENT_T10, "h27": xfem.ELEMENT_H27}.get(case.get("element"), 0)
    return dict(gravity=(0.0, 0.0, -9.81), compliance=compliance(case, young), poissons_ratio=case["nu"], flags=flags,
                yeoh=YEOH, ground=1 if case.get("ground") else 0, ground_normal=(0.0, 0.0, 1.0), friction=0.4,
                **damping_of(case))


def tagged(el):
    n = el.shape[1]
    return np.concatenate([np.full((len(el), 1), n), el], 1).astype(np.uint32).reshape(-1)


# ---- the calls ----------------------------------------------------------------
def pinned(n):
    return torch.empty(n, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    """The handle, stepped one frame so that its launch form is picked, then set
    to the case's state, and the arrays that results are read into."""
    inp = inputs(case, seed)
    b = xfem.Body(meshes=[(x.reshape(-1), tagged(el), DENSITY) for x, el, _ in inp["bodies"]],
                  settings=[settings_of(case, E, e) for E, e in zip(inp["young"], inp["energy"])])
    dt = FRAME / case["substeps"]
    if case["kind"] == "adjoint":
        b.set_tet_mu(inp["mu"])
        dt = 1.0 / 1200.0
    # the added nodes of quadratic elements start at the means of their corners: the handle has them
    x0 = [b.positions(i) for i in range(b.nbodies)]
    v0 = [v if len(x) == len(v) else velocity_of_all(case, b, v, i)
          for i, (x, (_, _, v)) in enumerate(zip(x0, inp["bodies"]))]
    if case["kind"] == "calls":
        b.substep(dt)
    else:
        b.step_frames(1, case["substeps"], dt)
    for i in range(b.nbodies):
        b.set_state(x0[i], v0[i], i)
    st = dict(body=b, case=case, dt=dt, nv=[len(x) for x in x0])
    if case["kind"] == "adjoint":
        st.update(x0=x0[0], v0=v0[0], **{k: inp[k] for k in ("mu", "tips", "target")})
    else:
        n = sum(st["nv"])
        st["x"], st["v"] = pinned(3 * n), pinned(3 * n)
    return st


def velocity_of_all(case, b, v, i):
    """Corner velocities carried to the added nodes (means of their corners)."""
    n = b.counts[i][0]
    out = np.zeros((n, 3), np.float32)
    out[:len(v)] = v
    if case["element"] == "t10":
        _, _, t10, edges = b.t10_rest_state(i)
        out[len(v):] = 0.5 * (v[edges[:, 0]] + v[edges[:, 1]])
    else:
        h27 = b.h27_rest_state(i)[2]
        corner, shape = h27[:, H27_CORNERS], h27_corner_weights()
        out[h27.reshape(-1)] = np.einsum("nc,ecd->end", shape, v[corner].astype(np.float64)).reshape(-1, 3)
        out[:len(v)] = v
    return out


def run(st):
    b, case = st["body"], st["case"]
    if case["kind"] == "adjoint":
        b.set_tet_mu(st["mu"])
        b.set_state(st["x0"], st["v0"])
        traj = b.adjoint_forward(case["substeps"], st["dt"], st["tips"])
        dmu, dx, dv = b.adjoint_backward(traj - st["target"])
        return {"trajectory": traj, "dmu": dmu, "dx": dx, "dv": dv}
    if case["kind"] == "calls":
        for _ in range(case["substeps"]):
            b.substep(st["dt"])
    else:
        b.step_frames(case.get("frames", 1), case["substeps"], st["dt"])
    o = 0
    for i, n in enumerate(st["nv"]):
        b.positions(i, out=st["x"][o:o + 3 * n])
        b.velocities(i, out=st["v"][o:o + 3 * n])
        o += 3 * n
    return {"x": st["x"].reshape(-1, 3), "v": st["v"].reshape(-1, 3)}


# ---- what a pass cannot do without ----------------------------------------------
def work(case):
    """A substep needs the whole of the one before it, so each reads every
    element's rest record and vertex ids and every vertex (position, velocity,
    inverse mass), and writes every vertex (position, velocity) once; the state
    goes to the host once per pass. The operations are those of one element
    solve (prefactored I1, the hydrostatic points, the 2x2 solve, the update)."""
    element = case.get("element", "tet")

    def flops(n, q):
        return 9 * n * (n - 1) + q * (36 * (n - 1) + 150) + 30 * n

    if case.get("bodies", 1) == 1:
        dims = [(case["w"], case["h"], case["d"])]
    else:  # the expected sizes
        dims = [tuple((2 + case[k]) / 2.0 for k in "whd")] * case["bodies"]
    nb = nf = nv = 0.0
    for w, h, d in dims:
        nc = w * h * d
        if element == "hex":
            v, ne, rec, f = (w + 1) * (h + 1) * (d + 1), nc, 160 + 32, flops(8, 1)
            if case["energy"] == "mixed":
                rec, f = 8 * 40 + 8 + 32, 8 * (36 * 7 * 2 + 200) + 30 * 8
        elif element == "h27":
            v, ne, rec, f = (2 * w + 1) * (2 * h + 1) * (2 * d + 1), nc, 4 * 432 + 108, flops(27, 8)
        else:
            ne = 6 * nc
            v, rec, f = (w + 1) * (h + 1) * (d + 1), 64 + 16, flops(4, 1)
            if element == "t10":
                v = v + 7 * nc + 3 * nc / min(w, h, d)  # about one node per edge
                rec, f = 224 + 40, flops(10, 4)
            if case["energy"] == "ring":
                f = 4 * 300
        nv += v
        nb += ne * rec + v * 52
        nf += ne * f + v * 30
    n = case["substeps"] * case.get("frames", 1)
    if case.get("damping") == "ui":
        nf *= 1.2  # an eighth of the elements damped twice
    if case["kind"] == "adjoint":
        # recording writes and the reverse pass reads a solve's inputs; the reverse does about twice the work
        nb, nf = 2 * nb + 2 * (48 * 6 * case["w"] * case["h"] * case["d"]), 3 * nf
    return {"bytes": n * nb + 24 * nv, "flops": n * nf}


# ---- the method in 64 bits --------------------------------------------------------
# Per substep: predict (gravity), then the elements in groups; the elements of a
# group share no vertex, and the groups follow the colour order that the
# documentation states (greedy colours in id order over cubes, edge stars,
# elements or one-rings). Then locks, ground with Coulomb friction, velocities.
H27_CORNERS = [0, 2, 6, 8, 18, 20, 24, 26]
HEX_EDGES = [(0, 1), (0, 2), (0, 4), (1, 3), (1, 5), (2, 3), (2, 6), (3, 7), (4, 5), (4, 6), (5, 7), (6, 7)]
HEX_FACES = [(0, 1, 3, 2), (4, 5, 7, 6), (0, 1, 5, 4), (2, 3, 7, 6), (0, 2, 6, 4), (1, 3, 7, 5)]
TET_EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


def h27_corner_weights():
    """Weights of the 8 corners at the 27 nodes of the 3x3x3 grid."""
    t = np.array([0.0, 0.5, 1.0])
    out = np.zeros((27, 8))
    for n in range(27):
        x = t[[n % 3, n // 3 % 3, n // 9]]
        for c in range(8):
            out[n, c] = np.prod([x[a] if c >> a & 1 else 1 - x[a] for a in range(3)])
    return out


def greedy(sets, n):
    """Colours in id order: the smallest that no earlier set sharing a member has."""
    mask = [0] * n
    out = []
    for s in sets:
        m = 0
        for v in s:
            m |= mask[v]
        c = (~m & (m + 1)).bit_length() - 1
        out.append(c)
        c = 1 << c
        for v in s:
            mask[v] |= c
    return np.array(out)


def edge_stars(tets):
    """Clusters in tet order: an unassigned tet takes the edge with the most
    unassigned tets (the first such) and those of its tets, in id order, that
    keep the cluster within 8 tets and 8 vertices."""
    around, ts = {}, tets.tolist()
    for t, q in enumerate(ts):
        for a, b in TET_EDGES:
            around.setdefault((min(q[a], q[b]), max(q[a], q[b])), []).append(t)
    free, out = [True] * len(ts), []
    for t, q in enumerate(ts):
        if not free[t]:
            continue
        best, count = None, 0
        for a, b in TET_EDGES:
            star = around[(min(q[a], q[b]), max(q[a], q[b]))]
            n = sum(free[k] for k in star)
            if n > count:
                best, count = star, n
        verts, got = [], []
        for k in best:
            if free[k] and len(got) < 8:
                more = verts + [v for v in ts[k] if v not in verts]
                if len(more) <= 8:
                    verts, free[k] = more, False
                    got.append(k)
        out.append((got, verts))
    return out


def tet_groups(case, el, w, h, d):
    """Tet ids of each group, in order."""
    nv = (w + 1) * (h + 1) * (d + 1)
    if case.get("mesh") != "shuffled":  # a cluster is a cube
        col = greedy(cubes(w, h, d).tolist(), nv)
        return [np.nonzero(col == c)[0] * 6 + t for c in range(col.max() + 1) for t in range(6)]
    cl = edge_stars(el)
    col = greedy([v for _, v in cl], nv)
    place = {}
    for (got, _), c in zip(cl, col):
        for k, t in enumerate(got):
            place.setdefault((int(c), k), []).append(t)
    return [np.array(place[k]) for k in sorted(place)]


def by_owner(lo, up, nv):
    """Distinct entries per lower vertex: in stream order, a later duplicate
    taking the list's last entry in its place. up: rows of ids. Returns the
    kept rows, vertex by vertex."""
    order = np.argsort(lo, kind="stable")
    off = np.searchsorted(lo[order], np.arange(nv + 1))
    seen, keep = {}, []
    rel = (up - lo[:, None])[order]
    same = np.sort(up, 1) if up.shape[1] > 1 else up
    same = (same - lo[:, None])[order]
    for v in range(nv):
        a, b = off[v], off[v + 1]
        if a == b:
            continue
        key = rel[a:b].tobytes()
        r = seen.get(key)
        if r is None:
            rows, L = [tuple(x) for x in same[a:b].tolist()], list(range(b - a))
            j = 0
            while j < len(L):
                k = j + 1
                while k < len(L):
                    if rows[L[j]] == rows[L[k]]:
                        last = L.pop()
                        if k < len(L):
                            L[k] = last
                    else:
                        k += 1
                j += 1
            r = seen[key] = np.array(L)
        keep.append(order[a + r])
    return np.concatenate(keep)


def find(keys, of):
    """Index in `keys` of each of `of`."""
    o = np.argsort(keys)
    return o[np.searchsorted(keys[o], of)]


def quadratic(el, nodes):
    """(elements with their added nodes, all positions): edges, faces, centres."""
    nv, x = len(nodes), nodes.astype(np.float64)
    pairs = TET_EDGES if el.shape[1] == 4 else HEX_EDGES
    inst = np.stack([el[:, list(p)] for p in pairs], 1).reshape(-1, 2)
    lo, up = inst.min(1), inst.max(1)
    keep = by_owner(lo, up[:, None], nv)
    edge_key = lo * nv + up
    ids = nv + find(edge_key[keep], edge_key).reshape(len(el), -1)
    xs = [x, 0.5 * (x[lo[keep]] + x[up[keep]])]
    if el.shape[1] == 4:
        return np.concatenate([el, ids], 1), np.concatenate(xs)
    ne = len(keep)
    face = np.stack([el[:, list(f)] for f in HEX_FACES], 1).reshape(-1, 4)
    r = face.argmin(1)
    face = face[np.arange(len(face))[:, None], (r[:, None] + np.arange(4)) % 4]
    keep = by_owner(face[:, 0], face[:, 1:], nv)
    face_key = face[:, 0] * nv + face[:, 2]
    fid = nv + ne + find(face_key[keep], face_key).reshape(len(el), -1)
    xs += [0.25 * x[face[keep]].sum(1), 0.125 * x[el].sum(1)]
    out = np.zeros((len(el), 27), np.int64)

    def node(cs):  # grid node at the mean of these corners
        i = sum(np.array([c & 1, c >> 1 & 1, c >> 2 & 1]) for c in cs) * 2 // len(cs)
        return i[0] + 3 * i[1] + 9 * i[2]

    for c in range(8):
        out[:, node([c])] = el[:, c]
    for k, p in enumerate(pairs):
        out[:, node(p)] = ids[:, k]
    for k, f in enumerate(HEX_FACES):
        out[:, node(f)] = fid[:, k]
    out[:, 13] = nv + ne + len(keep) + np.arange(len(el))
    return out, np.concatenate(xs)


def rules(element):
    """((gradients[Q, N, 3], weights[Q], corner gradients[Q, C, 3]) of the I1 rule and of the hydrostatic
    rule, corner columns, and the nodes' share of the mass or the shape values to form it from)."""
    if element in ("tet", "t10"):
        gl = np.array([[1.0, 0, 0], [0, 1, 0], [0, 0, 1], [-1, -1, -1]])
        if element == "tet":
            r = (gl[None], np.ones(1), gl[None])
            return r, r, [0, 1, 2, 3], np.full(4, 0.25)
        L = np.full((4, 4), (5 - math.sqrt(5)) / 20) + np.eye(4) * (math.sqrt(5) / 5)
        g = np.zeros((4, 10, 3))
        for p in range(4):
            for n in range(4):
                g[p, n] = (4 * L[p, n] - 1) * gl[n]
            for k, (a, b) in enumerate(TET_EDGES):
                g[p, 4 + k] = 4 * (L[p, b] * gl[a] + L[p, a] * gl[b])
        r = (g, np.full(4, 0.25), np.tile(gl, (4, 1, 1)))
        return r, r, [0, 1, 2, 3], np.array([13.0] * 4 + [70.0] * 6) / 472.0

    def shape(order, x):
        if order == 1:
            return np.array([(1 - x) / 2, (1 + x) / 2]), np.array([-0.5, 0.5])
        return np.array([x * (x - 1) / 2, 1 - x * x, x * (x + 1) / 2]), np.array([x - 0.5, -2 * x, x + 0.5])

    def table(order, pts):
        m = order + 1
        N, G = np.zeros((len(pts), m ** 3)), np.zeros((len(pts), m ** 3, 3))
        for p, x in enumerate(pts):
            f = [shape(order, v) for v in x]
            for n in range(m ** 3):
                i = (n % m, n // m % m, n // (m * m))
                N[p, n] = np.prod([f[a][0][i[a]] for a in range(3)])
                for k in range(3):
                    G[p, n, k] = np.prod([f[a][1 if a == k else 0][i[a]] for a in range(3)])
        return N, G

    def gauss(n):
        x, w = np.polynomial.legendre.leggauss(n)
        pts = [(x[i], x[j], x[k]) for k in range(n) for j in range(n) for i in range(n)]
        return np.array(pts), np.array([w[i] * w[j] * w[k] for k in range(n) for j in range(n) for i in range(n)])

    order, hi, lo = (1, 2, 1) if element == "hex" else (2, 3, 2)
    out = []
    for n in (hi, lo):
        pts, w = gauss(n)
        N, G = table(order, pts)
        out.append((G, w, table(1, pts)[1]))
        if n == hi:
            values = N
    return out[0], out[1], list(range(8)) if element == "hex" else H27_CORNERS, values


class Method:
    """The bodies of a case in one set of 64-bit arrays."""

    def __init__(self, case, inp, device):
        self.case, self.dev = case, device
        element = case.get("element", "tet")
        xs, vs, els, groups, first = [], [], [], {}, 0
        lock, mu, ne = [], [], 0
        for i, ((x, el, v), E) in enumerate(zip(inp["bodies"], inp["young"])):
            dims = (case["w"], case["h"], case["d"])
            if case.get("bodies", 1) > 1:  # the box's sides, from its cubes
                dims = sides(el)
            if element == "tet":
                gs = tet_groups(case, el, *dims)
            else:
                col = greedy(el.tolist(), len(x))
                gs = [np.nonzero(col == c)[0] for c in range(col.max() + 1)]
            pos = x.astype(np.float64)
            if element in ("t10", "h27"):
                corner_el = el
                el, pos = quadratic(el, x)
                vv = np.zeros((len(pos), 3))
                vv[:len(v)] = v
                if element == "t10":
                    for k, (a, b) in enumerate(TET_EDGES):
                        vv[el[:, 4 + k]] = 0.5 * (v[corner_el[:, a]].astype(np.float64) + v[corner_el[:, b]])
                else:
                    vv[el.reshape(-1)] = np.einsum("nc,ecd->end", h27_corner_weights(),
                                                   v[corner_el].astype(np.float64)).reshape(-1, 3)
                v = vv
            rel = (pos[:, 0] - x[:, 0].min()) / np.float64(x[:, 0].max() - x[:, 0].min())
            lock.append((rel < 0.02) & (not case.get("ground")))
            for k, g in enumerate(gs):
                groups.setdefault(k, []).append(g + ne)
            xs.append(pos)
            vs.append(v.astype(np.float64))
            els.append(el + first)
            mu.append(np.full(len(el), E / (4.0 * (1.0 + case["nu"]))))
            first += len(pos)
            ne += len(el)
        t = self.tensor
        self.x, self.v, self.el = t(np.concatenate(xs)), t(np.concatenate(vs)), t(np.concatenate(els))
        self.mu = t(inp["mu"].astype(np.float64) if "mu" in inp else np.concatenate(mu))
        self.groups = [t(np.concatenate(groups[k])) for k in sorted(groups)]
        yeoh = np.concatenate([np.full(len(e), float(m == "yeoh")) for e, m in zip(els, inp["energy"])])
        self.yeoh = t(yeoh)
        self.any_yeoh, self.any_nh = bool((yeoh > 0).any()), bool((yeoh == 0).any())
        self.ratio = 0.0 if case["nu"] >= 0.5 else (1.0 - 2.0 * case["nu"]) / (2.0 * case["nu"])
        self.a = 1.0 + self.ratio
        hi, lo, corners, mass = rules(element)
        if case["energy"] == "mixed":
            lo = hi
        P = self.x[self.el][:, corners]
        self.P = None
        (self.Bh, self.wh, _), (self.Bl, self.wl, vol) = self.mapped(P, hi), self.mapped(P, lo)
        if element in ("tet", "t10"):
            vol = torch.linalg.det(P[:, :3] - P[:, 3:]) / 6.0
        elif element == "hex":
            vol = self.mapped(P, hi)[2]
        self.vol = vol
        if element in ("hex", "h27"):
            N2 = t(mass * mass)
            m = self.wh @ N2
            share = m / m.sum(1, keepdim=True)
        else:
            share = t(np.tile(mass, (len(self.el), 1)))
        m = torch.zeros(len(self.x), dtype=torch.float64, device=device)
        m.index_add_(0, self.el.reshape(-1), (share * (DENSITY * vol)[:, None]).reshape(-1))
        self.w = torch.where(t(np.concatenate(lock)), torch.zeros_like(m), 1.0 / m)
        self.locked = t(np.concatenate(lock))[:, None]
        self.rings = self.ring_groups(case) if case["energy"] == "ring" else None

    def tensor(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def mapped(self, P, rule):
        """Gradients in the rest frame [E, Q, N, 3], normalised weights [E, Q], the volume of the rule."""
        G, w, M = (self.tensor(a) for a in rule)
        J = torch.einsum("qcr,ecd->eqdr", M, P)  # dX_d / dxi_r
        B = torch.einsum("qnr,eqrd->eqnd", G, torch.linalg.inv(J))
        w = torch.linalg.det(J) * w
        vol = w.sum(1)
        return B, w / vol[:, None], vol

    def deviatoric(self, I1, g, yeoh):
        """The energy's U0 and gradient from I1 and its gradient."""
        if self.case["energy"] == "mixed":
            return I1.clamp(min=1e-4), g
        if not self.any_yeoh:
            return I1, g
        s = I1 - 3.0
        U = (s * (YEOH[0] + s * (YEOH[1] + s * YEOH[2]))).clamp(min=1e-4)
        k = YEOH[0] + s * (2 * YEOH[1] + s * 3 * YEOH[2])
        if not self.any_nh:
            return U, g * k[:, None, None]
        y = yeoh > 0
        return torch.where(y, U, I1), torch.where(y[:, None, None], g * k[:, None, None], g)

    @staticmethod
    def cramer(A0, A1, A2, b0, b1):
        r0, r1 = A1 / A0, A1 / A2
        s = 1.0 / (1.0 - r0 * r1).clamp(min=1e-8)
        c0, c1 = b0 / A0, b1 / A2
        return s * (c0 - r0 * c1), s * (c1 - c0 * r1)

    def energies(self, X, e):
        """I1 and its gradient, (J - a)^2 and its gradient, of elements e at node positions X."""
        B, w = self.Bh[e], self.wh[e]
        P = X - X[:, -1:]
        F = torch.einsum("eki,eqka->eqia", P, B)
        I1 = (w * (F * F).sum((2, 3))).sum(1)
        g0 = 2.0 * torch.einsum("eq,eqia,eqka->eki", w, F, B)
        if self.Bl.shape[1] != self.Bh.shape[1] or self.Bl is not self.Bh:
            B, w = self.Bl[e], self.wl[e]
            F = torch.einsum("eki,eqka->eqia", P, B)
        a, b, c = F[..., 0], F[..., 1], F[..., 2]
        bc = torch.linalg.cross(b, c)
        J = (a * bc).sum(-1)
        cof = torch.stack([bc, torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -1)
        U1 = (w * (J - self.a) ** 2).sum(1)
        g1 = 2.0 * torch.einsum("eq,eqia,eqka->eki", w * (J - self.a), cof, B)
        return I1, g0, U1, g1

    def solve(self, O, D, w, e, dt, mu):
        n = self.el[e]
        wn = w[n]
        I1, g0, U1, g1 = self.energies(O[n] + D[n], e)
        U0, g0 = self.deviatoric(I1, g0, self.yeoh[e])
        alpha0 = 1.0 / (mu[e] * self.vol[e] * dt * dt)
        alpha1 = alpha0 * self.ratio
        A0 = 2 * U0 * alpha0 + 1e-22 + (wn * (g0 * g0).sum(2)).sum(1)
        A1 = 1e-22 + (wn * (g0 * g1).sum(2)).sum(1)
        A2 = 2 * U1 * alpha1 + 1e-22 + (wn * (g1 * g1).sum(2)).sum(1)
        l0, l1 = self.cramer(A0, A1, A2, -2 * U0, -2 * U1)
        step = wn[..., None] * (l0[:, None, None] * g0 + l1[:, None, None] * g1)
        return D.index_add(0, n.reshape(-1), step.reshape(-1, 3))

    def ring_groups(self, case):
        """Per ring colour: the vertices that are centres, and the tets around them."""
        el = self.el.cpu().numpy()
        nv = len(self.x)
        nodes = [set() for _ in range(nv)]
        for q in el.tolist():
            for v in q:
                nodes[v].update(q)
        col = greedy(nodes, nv)
        vert, tet = el.reshape(-1), np.repeat(np.arange(len(el)), 4)
        out = []
        for c in range(col.max() + 1):
            m = col[vert] == c
            out.append((self.tensor(vert[m]), self.tensor(tet[m])))
        return out

    def solve_rings(self, O, D, w, group, dt):
        centre, t = group  # the rings of a colour share no node: one sum per vertex is one ring's
        nv = len(O)
        n = self.el[t]

        def ring_sum(x):
            return torch.zeros(nv, dtype=x.dtype, device=x.device).index_add(0, centre, x)

        share = 0.25 * self.vol[t]
        vol = ring_sum(share)
        ew = share / vol[centre]
        X = O[n] + D[n]
        P = X[:, :3] - X[:, 3:]
        B, Q = self.Bh[t][:, 0], P
        F = torch.einsum("eki,eka->eia", Q, B[:, :3])
        I1 = ring_sum(ew * (F * F).sum((1, 2)))
        gI = 2.0 * torch.einsum("eia,eka->eki", F, B)
        a, b, c = F[..., 0], F[..., 1], F[..., 2]
        bc = torch.linalg.cross(b, c)
        J = ring_sum(ew * (a * bc).sum(-1))
        cof = torch.stack([bc, torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -1)
        gJ = torch.einsum("eia,eka->eki", cof, B)
        flat = n.reshape(-1)
        g0 = torch.zeros_like(O).index_add(0, flat, (ew[:, None, None] * gI).reshape(-1, 3))
        g1 = torch.zeros_like(O).index_add(0, flat, (ew[:, None, None] * gJ).reshape(-1, 3))
        ring = torch.zeros(nv, dtype=torch.int64, device=O.device)
        ring[flat] = centre[:, None].expand(-1, 4).reshape(-1)
        g1 = g1 * (2.0 * (J - self.a))[ring][:, None]
        touched = torch.unique(flat)

        def wsum(x, y):
            v = w[touched] * (x[touched] * y[touched]).sum(1)
            return 1e-22 + torch.zeros(nv, dtype=v.dtype, device=v.device).index_add(0, ring[touched], v)

        mu = self.mu[0]
        on = torch.unique(centre)
        U0, U1 = I1[on], (J[on] - self.a) ** 2
        alpha0 = 1.0 / (mu * vol[on] * dt * dt)
        l0, l1 = self.cramer(2 * U0 * alpha0 + wsum(g0, g0)[on], wsum(g0, g1)[on],
                             2 * U1 * alpha0 * self.ratio + wsum(g1, g1)[on], -2 * U0, -2 * U1)
        L0 = torch.zeros(nv, dtype=O.dtype, device=O.device).index_copy(0, on, l0)
        L1 = torch.zeros(nv, dtype=O.dtype, device=O.device).index_copy(0, on, l1)
        step = w[touched, None] * (L0[ring[touched], None] * g0[touched] + L1[ring[touched], None] * g1[touched])
        return D.index_add(0, touched, step)

    def contact(self, O, D):
        depth = -(O[:, 2] + D[:, 2])
        hit = (depth > 0) & (self.w > 0)
        lift = torch.where(hit, depth, torch.zeros_like(depth))
        D = torch.stack([D[:, 0], D[:, 1], D[:, 2] + lift], 1)
        lt = torch.sqrt(D[:, 0] ** 2 + D[:, 1] ** 2)
        lim = 0.4 * lift
        s = torch.where(lt <= lim, torch.ones_like(lt), lim / lt)
        keep = torch.where(hit, 1.0 - s, torch.ones_like(s))
        return torch.stack([D[:, 0] * keep, D[:, 1] * keep, D[:, 2]], 1)

    def substep(self, X, V, dt, mu):
        g = torch.tensor([0.0, 0.0, -9.81], dtype=torch.float64, device=X.device)
        D = (V + g * dt) * dt
        if self.rings:
            for r in self.rings:
                D = self.solve_rings(X, D, self.w, r, dt)
        else:
            for e in self.groups:
                D = self.solve(X, D, self.w, e, dt, mu)
        D = torch.where(self.locked, torch.zeros_like(D), D)
        if self.case.get("ground"):
            D = self.contact(X, D)
        return X + D, D / dt


def sides(el):
    """(w, h, d) of a box from its tets: the first cube's corners give the strides."""
    c = el[0].min()
    corner = np.unique(el[:6])
    sx, sxy = int(corner[2] - c), int(corner[4] - c)
    n = len(el) // 6
    w = sx - 1
    h = sxy // sx - 1
    return w, h, n // (w * h)


def exact(case, seed):
    """run()'s first pass in 64 bits. None where the eighth of the elements that a
    substep damps is the handle's own choice, where it would take long, and for
    the velocities of an incompressible material: its multiplier goes as
    1 / (J - 1), so 32 bits say little about them."""
    n = case["substeps"] * case.get("frames", 1)
    elements = work(case)["flops"] / n
    if case.get("damping") == "ui" or (case["kind"] == "adjoint" and (elements > 3e7 or n > 200)):
        return None
    if case.get("mesh") == "shuffled" and case["w"] * case["h"] * case["d"] > 14000:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    inp = inputs(case, seed)
    if case["kind"] == "adjoint":
        return exact_gradient(case, inp)
    with torch.no_grad():
        m = Method(case, inp, device)
        X, V = m.x, m.v
        for _ in range(n):
            X, V = m.substep(X, V, FRAME / case["substeps"], m.mu)
    return {"x": X.cpu().numpy(), "v": None if case["nu"] >= 0.5 else V.cpu().numpy()}


def exact_gradient(case, inp):
    m = Method(case, inp, "cpu")  # some thousand tets: the launches would cost more than the work
    X, V, mu = (t.clone().requires_grad_(True) for t in (m.x, m.v, m.mu))
    tips = torch.from_numpy(inp["tips"].astype(np.int64))
    x, v, traj = X, V, []
    for _ in range(case["substeps"]):
        x, v = m.substep(x, v, 1.0 / 1200.0, mu)
        traj.append(x[tips])
    traj = torch.stack(traj)
    cot = (traj - torch.from_numpy(inp["target"].astype(np.float64))).detach()
    dmu, dx, dv = torch.autograd.grad(traj, (mu, X, V), cot)
    return {"trajectory": traj.detach().numpy(), "dmu": dmu.numpy(), "dx": dx.numpy(), "dv": dv.numpy()}
