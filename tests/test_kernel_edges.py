"""Kernels at the sizes where their tiling can go wrong: edges of tiles,
remainders, the smallest and largest of a dispatch rule's range."""

import ctypes as C

import numpy as np
import pytest

import kat_scenes as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [4, 5, 18, 33])
@pytest.mark.parametrize("mesh", ["cube", "sphere6x5", "torus21x11", "far", "nan"])
def test_bake_bricks_and_chunks(oracle, res, mesh):
    """Grids that are no multiple of a warp's brick against meshes of one
    chunk of triangles, a partial last chunk, far from the origin, and with a
    triangle whose corner is not a number: the oracle's field bit for bit."""
    from pfsim import mesh as M

    if mesh == "sphere6x5":
        v, i = K.uv_sphere(0.5, 6, 5)
    elif mesh == "torus21x11":
        v, i = K.torus(0.4, 0.12, 21, 11)
    else:
        v, i = K.unit_cube_mesh((0.3, 0.2, 0.45))
        if mesh == "far":
            v = (v + np.array([37.0, -5.0, 110.0], np.float32)).astype(np.float32)
        elif mesh == "nan":
            v = np.vstack([v, np.array([[np.nan, 0.0, 0.0]], np.float32)])
            i = np.concatenate([i, np.array([0, 1, len(v) - 1], np.uint32)])
    a = M.bake_sdf(v, i, res, 0.07)
    b = oracle.bake_sdf(v, i, res, 0.07)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2] and a[3] == b[3]


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
def test_readback_in_particle_order(oracle, n):
    """Every per-slot field of a scene that ends on, before and after a
    256-slot block, after a step that reorders the slots: the oracle's, row
    for row (particles of no fluid read as zero density and multiplier)."""
    from pfsim import _native as N
    from pfsim import recipe as R

    r = np.random.default_rng(n)
    pos = r.uniform(0.2, 0.5, (n, 3)).astype(np.float32)
    half = max(1, n // 2)
    rec = R.Recipe(capacity=n, radius=0.01, uploads=[R.Upload(0, pos, r.normal(0, 0.1, (n, 3)).astype(np.float32))],
                   materials=[("fluid", R.FluidOpts(range=(0, half), particle_spacing=0.02, rest_density=1000.0,
                                                    viscosity=0.01))],
                   prims=R.container_walls((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)), loop=R.LoopOpts(substeps=1, iterations=2))
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    a.step(1 / 60)
    b.step(1 / 60)
    for f in (N.PF_FIELD_POSITIONS, N.PF_FIELD_PREDICTED, N.PF_FIELD_VELOCITIES, N.PF_FIELD_INV_MASS,
              N.PF_FIELD_BOUNDARY_VOLUME, N.PF_FIELD_DENSITY):
        x, y = a.readback(f), b.readback(f)
        assert x.shape == y.shape
        # single precision against single precision over one substep: sums of
        # at most 64 terms, each rounded to 2^-24, and one division by dt
        assert np.allclose(x, y, rtol=1e-4, atol=1e-4), f
    assert not a.readback(N.PF_FIELD_DENSITY)[half:].any() and not a.readback(N.PF_FIELD_LAMBDA)[half:].any()
    a.close()


@pytest.mark.parametrize("substeps", [1, 2, 3])
def test_plain_steps_as_graph_same_bits(pfsim, substeps):
    """A plain scene's steps are launched one by one at first and as a graph
    later: the same bits throughout as the same scene stepped without graphs,
    for odd and even substeps (one or two start parities), across a moving
    collider and a mass write that changes what is launched."""
    from pfsim import _native as N
    from pfsim import recipe as R
    from pfsim import workloads as W

    rec = W.dam_break(3000, seed=substeps, substeps=substeps, iterations=2)
    rec.prims.append(R.sphere((0.2, 0.1, 0.0), 0.08))
    a = R.NativeBackend().build(rec)
    b = R.Batch([R.NativeBackend().build(rec)], use_graph=False)
    for k in range(10):
        if k == 6:  # after the capture
            w = np.linspace(0.9, 1.1, rec.capacity).astype(np.float32) * a.readback(N.PF_FIELD_INV_MASS)
            a.write(N.PF_FIELD_INV_MASS, w)
            b.write(0, N.PF_FIELD_INV_MASS, w)
        q = R.sphere((0.2 - 0.01 * k, 0.1, 0.0), 0.08, velocity=(-0.6, 0.0, 0.0))
        a.set_primitive(len(rec.prims) - 1, q)
        p = q.cstruct()
        N.check(N.lib().pf_batch_set_primitive(b.h, 0, len(rec.prims) - 1, C.byref(p)))
        a.step(1 / 60)
        b.step(1 / 60)
        for f in (N.PF_FIELD_POSITIONS, N.PF_FIELD_VELOCITIES):
            assert np.array_equal(a.readback(f), b.readback(0, f)), k
    a.close()
    b.close()


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("unroll", [2, 4, 8])
@pytest.mark.parametrize("per_cell", [1, 3, 8, 30, 70])
def test_list_build_columns(oracle, monkeypatch, per_cell, unroll, wide):
    """The neighbour list where a lane's column of hits stays nearly empty, is
    filled in the last rows, and overflows (64 entries at most, the rest
    flagged), with 16- and 32-bit entries: the oracle's lists, element for
    element."""
    from pfsim import _native as N
    from pfsim import recipe as R

    monkeypatch.setenv("PFSIM_NBR_PATH", "0")
    monkeypatch.setenv("PFSIM_SLOT_BLOCK", "128")
    monkeypatch.setenv("PFSIM_SLOT_UNROLL", str(unroll))
    monkeypatch.setenv("PFSIM_NBR_WIDE", str(wide))
    h = 0.04
    r = np.random.default_rng(per_cell)
    n = 125 * per_cell + 7
    pos = r.uniform(0.2, 0.2 + 5 * h, (n, 3)).astype(np.float32)
    rec = R.Recipe(capacity=n, radius=0.005, uploads=[R.Upload(0, pos)],
                   materials=[("fluid", R.FluidOpts(range=(0, n), particle_spacing=0.02, smoothing_radius=h,
                                                    rest_density=1000.0, viscosity=0.01))],
                   loop=R.LoopOpts(substeps=1, iterations=1, gravity=(0.0, 0.0, 0.0)))
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    a.step(1 / 60)
    b.step(1 / 60)
    for f in (N.PF_FIELD_NEIGHBOR_COUNT, N.PF_FIELD_NEIGHBORS):
        assert np.array_equal(a.readback(f), b.readback(f))
    assert a.overflow()["neighbors"] == b.overflow()["neighbors"] == (per_cell == 70 or per_cell == 30)
    # densities: sums of at most 64 positive terms, each rounded a few times
    np.testing.assert_allclose(a.readback(N.PF_FIELD_DENSITY), b.readback(N.PF_FIELD_DENSITY), rtol=2e-5)
    a.close()


@pytest.mark.parametrize("case", ["one", "overflow", "two_fluids", "boundary"])
@pytest.mark.parametrize("unroll", [2, 4, 8])
def test_surface_impulses_gathered_or_scattered(oracle, monkeypatch, case, unroll):
    """Surface tension and adhesion where every particle gathers its own
    changes (one fluid, with and without boundary particles) and where pairs
    are scattered (an overflowing list; two fluids): the oracle's positions
    and velocities."""
    from pfsim import _native as N
    from pfsim import recipe as R

    monkeypatch.setenv("PFSIM_NBR_PATH", "0")
    monkeypatch.setenv("PFSIM_SLOT_BLOCK", "128")
    monkeypatch.setenv("PFSIM_SLOT_UNROLL", str(unroll))
    s = 0.02
    g = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3) * s
    r = np.random.default_rng(unroll)
    pos = (0.3 + g + r.uniform(-0.1 * s, 0.1 * s, g.shape)).astype(np.float32)
    if case == "overflow":  # 90 particles in one cell's reach
        pos[:90] = (0.3 + r.uniform(0, 0.6 * s, (90, 3))).astype(np.float32)
    n, m = len(pos), len(pos) // 2
    opts = dict(rest_density=1000.0, particle_spacing=s, smoothing_radius=2 * s, viscosity=0.01, surface_tension=0.1,
                adhesion=0.1)
    if case == "two_fluids":
        mats = [("fluid", R.FluidOpts(range=(0, m), **opts)), ("fluid", R.FluidOpts(range=(m, n - m), **opts))]
    elif case == "boundary":
        mats = [("fluid", R.FluidOpts(range=(0, m), boundaries=[(m, n - m)], boundary_static=[True], **opts))]
    else:
        mats = [("fluid", R.FluidOpts(range=(0, n), **opts))]
    w = None
    if case == "boundary":
        w = np.zeros(n, np.float32)
    rec = R.Recipe(capacity=n, radius=s / 2, uploads=[R.Upload(0, pos, None, w)], materials=mats,
                   loop=R.LoopOpts(substeps=2, iterations=2))
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    a.step(1 / 120)
    b.step(1 / 120)
    # (the oracle's flag is the last substep's list's, the scene's the frame's)
    assert a.overflow()["neighbors"] == (case == "overflow")
    x, y = a.readback(N.PF_FIELD_POSITIONS), b.readback(N.PF_FIELD_POSITIONS)
    # 1e-5 of the block's 0.18 m would be 1.8e-6; the clump of `overflow`
    # is pushed apart by metres per second, so its bound is relative to that
    tol = 2e-6 if case != "overflow" else 1e-4 * max(1.0, float(np.abs(y).max()))
    assert np.abs(x - y).max() <= tol
    a.close()


@pytest.mark.parametrize("n", [1, 33, 1_023, 16_384, 16_385, 32_769, 65_536, 65_537])
@pytest.mark.parametrize("dims", [(2, 1, 1), (16, 16, 1), (17, 16, 1), (64, 64, 64), (64, 64, 65), (200, 100, 100)])
def test_sort_in_one_cluster(oracle, n, dims):
    """The sort of few elements in one thread-block cluster and its limits:
    one to four elements a thread, one to three passes, cell counts scanned in
    the cluster or after it; spread over the grid, and half of them in one
    cell. The oracle's keys, counts, starts and permutation."""
    from pfsim import hashgrid as H

    r = np.random.default_rng(n + dims[0])
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = r.uniform(0.0, 1.0, (n, 3)) * np.array(dims) * 0.1
    pos[: n // 2, :3] = pos[n - 1, :3]
    g = H.GridOptions(cell_size=0.1, kind="linear", dims=dims)
    a, b = H.sort(pos, g), oracle.sort(pos, g.desc(n))
    assert np.array_equal(a.cell_index, b["keys"])
    assert np.array_equal(a.counts, b["count"])
    assert np.array_equal(a.cell_start, b["start"])
    assert np.array_equal(a.sorted_indices, b["perm"])


@pytest.mark.parametrize("edges", ["lattice", "star", "complete", "pair"])
@pytest.mark.parametrize("fluid", [False, True])
def test_cluster_layouts(oracle, edges, fluid):
    """Shape matching over clusters of equal size, one large cluster among
    small ones (a warp's lists laid out cluster after cluster), every particle
    in every cluster, and particles without neighbours; in a world without a
    grid and in one whose slots move (a fluid beside the body): the oracle's
    positions and orientations."""
    from pfsim import _native as N
    from pfsim import recipe as R

    g = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.02 + [0.3, 0.02, 0.3]
    n = 70 if edges == "complete" else 125
    g = g[:n]
    if edges == "lattice":
        d = np.abs(g[:, None] - g[None]).max(-1)
        e = np.argwhere((d < 0.025) & (np.arange(n)[:, None] < np.arange(n)[None]))
    elif edges == "star":
        e = np.array([(0, k) for k in range(1, n)])
    elif edges == "complete":
        e = np.array([(i, j) for i in range(n) for j in range(i + 1, n)])
    else:
        e = np.array([(0, 1)])
    r = np.random.default_rng(3)
    pos = g.astype(np.float32)
    vel = r.normal(0, 0.2, (n, 3)).astype(np.float32)
    w = np.full(n, 1.0 / 0.008, np.float32)
    ups, mats = [R.Upload(0, pos, vel, w)], [("soft", R.SoftbodyOpts([R.BodyDef(
        range=(0, n), compliance=1e-5, edges=e.astype(np.uint32))], "local"))]
    cap = n
    if fluid:
        f = (r.uniform(0, 0.1, (300, 3)) + [0.6, 0.05, 0.3]).astype(np.float32)
        ups.append(R.Upload(n, f))
        mats.append(("fluid", R.FluidOpts(range=(n, 300), particle_spacing=0.02, rest_density=1000.0, viscosity=0.01)))
        cap += 300
    rec = R.Recipe(capacity=cap, radius=0.01, uploads=ups, materials=mats,
                   prims=R.container_walls((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)), loop=R.LoopOpts(substeps=2, iterations=3))
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    a.step(1 / 60)
    b.step(1 / 60)
    # positions within 1e-5 of the container's metre; quaternions of unit
    # length, from rotations of clusters a few centimetres wide: 1e-5 / 0.02
    x, y = a.readback(N.PF_FIELD_POSITIONS)[:n], b.readback(N.PF_FIELD_POSITIONS)[:n]
    assert np.abs(x - y).max() <= 1e-5
    q, p = a.readback(N.PF_FIELD_ROTATION)[:n], b.readback(N.PF_FIELD_ROTATION)[:n]
    assert np.abs(q - p).max() <= 5e-4
    a.close()


@pytest.mark.parametrize("side", [2, 3, 12, 46])
@pytest.mark.parametrize("fluid", [False, True])
def test_cloth_colours_in_a_chain(oracle, side, fluid):
    """Sheets whose colours hold one constraint, less than a block and a few
    blocks, with bending and tethers, alone and beside a fluid whose grid
    moves the slots between substeps: the oracle's positions within 1e-5 of
    the container."""
    from pfsim import _native as N
    from pfsim import recipe as R
    from pfsim import workloads as W

    rec = W.cloth_sheet(side, seed=3, bend_compliance=1e-5, tethers=True, stretch_tolerance=0.06, wind=(0.8, 0.0, 1.5))
    n = rec.capacity
    if fluid:
        r = np.random.default_rng(5)
        f = (r.uniform(0, 0.1, (300, 3)) + [0.3, 0.05, 0.3]).astype(np.float32)
        rec.uploads.append(R.Upload(n, f))
        rec.materials.append(("fluid", R.FluidOpts(range=(n, 300), particle_spacing=0.02, rest_density=1000.0,
                                                   viscosity=0.01)))
        rec.capacity = n + 300
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    a.step(1 / 60)
    b.step(1 / 60)
    x, y = a.readback(N.PF_FIELD_POSITIONS)[:n], b.readback(N.PF_FIELD_POSITIONS)[:n]
    assert np.abs(x - y).max() <= 1e-5
    a.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 3000])
@pytest.mark.parametrize("quiet", [False, True])
def test_contact_lanes(oracle, n, quiet):
    """Crowded particles, so that rows hold more candidates and slots more
    pairs than a slot has lanes, with collision groups, pinned particles and,
    in half the worlds, a range that emits no pairs: the oracle's pairs, and
    its positions within 1e-5 of the box after the pairs' solve."""
    from pfsim import _native as N
    from pfsim import recipe as R

    r, rng = 0.02, np.random.default_rng(7 * n + quiet)
    side = (n * 4.19 * (2.2 * r) ** 3 / 16) ** (1 / 3)  # sixteen particles in reach of one
    pos = rng.uniform(0, side, (n, 3)).astype(np.float32)
    rec = K.particles(pos, r, 1, 2, gravity=(0, 0, 0), inv_mass=(rng.random(n) > 0.2).astype(np.float32),
                      group=rng.integers(0, 4, n), contact=(64 * n, 0.5, 0.4),
                      quiet=[(n // 4, n // 4)] if quiet and n >= 4 else [])
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend(precision=32).build(rec)
    a.step(K.DT)
    b.step(K.DT)
    (ca, pa), (cb, pb) = a.contacts(), b.contacts()
    assert ca == cb and {tuple(p) for p in pa.tolist()} == {tuple(p) for p in pb.tolist()}
    x, y = a.readback(N.PF_FIELD_POSITIONS)[:, :3], b.readback(N.PF_FIELD_POSITIONS)[:, :3]
    assert np.abs(x - y).max() <= 1e-5 * max(1.0, side)
    a.close()


@pytest.mark.parametrize("m", [1, 15, 33, 600])
@pytest.mark.parametrize("static", [True, False])
def test_boundary_volume_lanes(oracle, m, static):
    """Boundaries of one particle up to several hundred in a few cells, so
    that a row holds less than one round of a slot's lanes, and several: the
    oracle's volumes within 64 float roundings (a sum of some hundred
    positive terms and one quotient)."""
    from pfsim import _native as N
    from pfsim import recipe as R

    rng, s, nf = np.random.default_rng(m), 0.02, 64
    f = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * s + [0.3, 0.3, 0.3]
    b = rng.uniform(0, 0.08, (m, 3)) + [0.3, 0.2, 0.3]
    pos = np.concatenate([f, b]).astype(np.float32)
    rec = R.Recipe(capacity=nf + m, radius=0.01,
                   uploads=[R.Upload(0, pos, np.zeros_like(pos), np.r_[np.full(nf, 125.0), np.zeros(m)].astype(np.float32))],
                   materials=[("fluid", R.FluidOpts(range=(0, nf), particle_spacing=s, rest_density=1000.0,
                                                    viscosity=0.01, boundaries=[(nf, m)], boundary_static=[static]))],
                   prims=R.container_walls((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)),
                   loop=R.LoopOpts(substeps=1, iterations=2))
    a, o = R.NativeBackend().build(rec), oracle.OracleBackend(precision=32).build(rec)
    a.step(1 / 60)
    o.step(1 / 60)
    x, y = (w.readback(N.PF_FIELD_BOUNDARY_VOLUME)[nf:].astype(np.float64) for w in (a, o))
    assert (y > 0).all() and (np.abs(x - y) <= 64 * 2.0**-23 * y).all()
    a.close()


@pytest.mark.parametrize("blocks", [0, 8])
def test_sort_where_the_cluster_cannot_be_placed(blocks):
    """A device that places no 16-block cluster takes one of 8 blocks (half the
    elements at most), or none and the separate passes: the stable order on
    both sides of every line, in a process of its own (the choice is made
    once)."""
    import os
    import subprocess
    import sys

    from conftest import PKG

    code = """
import numpy as np
from pfsim import hashgrid as H
for n in (1, 8191, 8193, 16384, 16385, 32768, 32769, 65536, 65537):
    for dims in ((16, 16, 1), (64, 64, 65)):
        r = np.random.default_rng(n)
        pos = np.zeros((n, 4), np.float32)
        pos[:, :3] = r.uniform(0.0, 1.0, (n, 3)) * np.array(dims) * 0.1
        pos[: n // 2, :3] = pos[n - 1, :3]
        a = H.sort(pos, H.GridOptions(cell_size=0.1, kind="linear", dims=dims))
        assert np.array_equal(a.sorted_indices, np.argsort(a.cell_index, kind="stable")), (n, dims)
        count = np.bincount(a.cell_index, minlength=int(np.prod(dims)))
        assert np.array_equal(a.counts, count) and np.array_equal(a.cell_start, np.cumsum(count) - count), (n, dims)
"""
    env = dict(os.environ, PYTHONPATH=str(PKG), PFSIM_SORT_CLUSTER=str(blocks))
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


def _lattice_body(k, offset, spin):
    """A k^3 lattice of 2 cm spacing with edges between near points, spinning."""
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.02
    d = np.abs(g[:, None] - g[None]).max(-1)
    e = np.argwhere((d < 0.025) & (np.arange(len(g))[:, None] < np.arange(len(g))[None]))
    return (g + offset).astype(np.float32), np.cross(spin, g - g.mean(0)).astype(np.float32), e.astype(np.uint32)


def _chain_edges(n):
    return np.stack([np.arange(n - 1), np.arange(1, n)], 1).astype(np.uint32)


@pytest.mark.parametrize("second", ["local", "global"])
@pytest.mark.parametrize("case", ["apart", "around", "around_reversed", "shared", "part_shared"])
def test_two_softbody_systems(oracle, case, second):
    """Two soft-body systems in one scene: one after the other, one whose
    bodies lie on both sides of the other's, and over the same particles (all
    or some of them) with clusters and rest shapes of their own: the oracle's
    positions and orientations after two frames."""
    from pfsim import _native as N
    from pfsim import recipe as R

    spin = np.array([6.0, -9.0, 4.0])
    parts = [_lattice_body(k, [0.2 + 0.25 * b, 0.4, 0.3], spin) for b, k in enumerate((3, 4, 3))]
    first = np.cumsum([0] + [len(p[0]) for p in parts])
    pos, vel = np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    n = len(pos)

    def body(b, edges=None, scale=1.0, compliance=1e-5):
        rest = parts[b][0] * np.float32(scale)
        return R.BodyDef(range=(int(first[b]), len(parts[b][0])), compliance=compliance, rest_positions=rest,
                         edges=parts[b][2] if edges is None else edges)

    if case == "apart":
        a, b = [body(0)], [body(1), body(2)]
    elif case.startswith("around"):
        a, b = [body(0), body(2)], [body(1)]
    elif case == "shared":
        a, b = [body(0), body(1)], [body(0, _chain_edges(27), 1.02, 1e-4), body(1, scale=0.99)]
    else:
        a, b = [body(0), body(1)], [body(1, _chain_edges(64), 1.01, 1e-4), body(2)]
    mats = [("soft", R.SoftbodyOpts(a, "local")), ("soft", R.SoftbodyOpts(b, second))]
    if case == "around_reversed":
        mats.reverse()
    rec = R.Recipe(capacity=n, radius=0.01, uploads=[R.Upload(0, pos, vel, np.full(n, 125.0, np.float32))],
                   materials=mats, prims=R.container_walls((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)),
                   loop=R.LoopOpts(substeps=2, iterations=3))
    s, o = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    for _ in range(2):
        s.step(1 / 60)
        o.step(1 / 60)
    # positions within 1e-5 of the container's metre a frame; quaternions of
    # unit length, from rotations of clusters a few centimetres wide
    x, y = s.readback(N.PF_FIELD_POSITIONS), o.readback(N.PF_FIELD_POSITIONS)
    assert np.abs(x - y).max() <= 2e-5
    q, p = s.readback(N.PF_FIELD_ROTATION), o.readback(N.PF_FIELD_ROTATION)
    assert np.abs(q - p).max() <= 1e-3
    s.close()


def test_softbodies_of_a_batch_at_different_ranks(pfsim):
    """Scenes whose soft bodies are their first and their second material, in
    one batch: the positions, orientations and so the spins of the scenes
    stepped alone."""
    from pfsim import _native as N
    from pfsim import recipe as R

    recs = []
    for fluid_first in (False, True):
        x, v, e = _lattice_body(4, [0.3, 0.4, 0.3], np.array([8.0, -5.0, 3.0]))
        ups, mats = [R.Upload(0, x, v, np.full(64, 125.0, np.float32))], []
        soft = ("soft", R.SoftbodyOpts([R.BodyDef(range=(0, 64), compliance=1e-5, edges=_chain_edges(64))], "local"))
        if fluid_first:
            f = (np.random.default_rng(4).uniform(0, 0.1, (200, 3)) + [0.6, 0.05, 0.3]).astype(np.float32)
            ups.append(R.Upload(64, f))
            mats.append(("fluid", R.FluidOpts(range=(64, 200), particle_spacing=0.02, rest_density=1000.0,
                                              viscosity=0.01)))
        mats.append(soft)
        recs.append(R.Recipe(capacity=264 if fluid_first else 64, radius=0.01, uploads=ups, materials=mats,
                             prims=R.container_walls((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)),
                             loop=R.LoopOpts(substeps=2, iterations=2)))
    alone = [R.NativeBackend().build(r) for r in recs]
    batch = R.Batch([R.NativeBackend().build(r) for r in recs])
    for _ in range(3):
        batch.step(1 / 60)
        for s in alone:
            s.step(1 / 60)
    for i, s in enumerate(alone):
        for f in (N.PF_FIELD_POSITIONS, N.PF_FIELD_ROTATION):
            assert np.array_equal(s.readback(f)[:64], batch.readback(i, f)[:64]), (i, f)
    batch.close()


def _two_fluids_on_one_slab(a_bnd, b_bnd):
    """Two fluids side by side on a slab of free particles, each with its own
    range of the slab as a dynamic boundary."""
    from pfsim import recipe as R

    s = 0.02
    fluid = np.stack(np.meshgrid(np.arange(4), np.arange(4), np.arange(8), indexing="ij"), -1).reshape(-1, 3) * s
    slab = np.stack(np.meshgrid(np.arange(8), np.arange(2), np.arange(8), indexing="ij"), -1).reshape(-1, 3) * s
    r = np.random.default_rng(11)
    pos = np.concatenate([fluid + [0.3, 0.34, 0.3], fluid + [0.38, 0.34, 0.3], slab + [0.3, 0.3, 0.3]])
    pos = (pos + r.uniform(-0.1 * s, 0.1 * s, pos.shape)).astype(np.float32)
    opts = dict(particle_spacing=s, smoothing_radius=2 * s, rest_density=1000.0, viscosity=0.01)
    mats = [("fluid", R.FluidOpts(range=(128 * k, 128), boundaries=[(256 + b, n) for b, n in bnd],
                                  boundary_static=[False] * len(bnd), **opts)) for k, bnd in enumerate((a_bnd, b_bnd))]
    return R.Recipe(capacity=384, radius=0.01, uploads=[R.Upload(0, pos, None, np.full(384, 125.0, np.float32))],
                    materials=mats, prims=R.container_walls((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)),
                    loop=R.LoopOpts(substeps=2, iterations=3))


@pytest.mark.parametrize("b_bnd", [[(32, 96)], [(64, 64), (0, 48)], []])
@pytest.mark.parametrize("a_bnd", [[(0, 96)], [(16, 16), (40, 60)]])
def test_reactions_on_a_boundary_of_two_fluids(oracle, nbr_path, a_bnd, b_bnd):
    """Slab particles on one fluid's boundary, on both fluids' (their tag
    names the second fluid's, so the first one's ranges are searched), and on
    none: the oracle's positions within 1e-5 of the box, from reactions that
    move the slab by much more than that."""
    from pfsim import _native as N
    from pfsim import recipe as R

    rec = _two_fluids_on_one_slab(a_bnd, b_bnd)
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend().build(rec)
    a.step(1 / 60)
    b.step(1 / 60)
    x, y = a.readback(N.PF_FIELD_POSITIONS), b.readback(N.PF_FIELD_POSITIONS)
    assert np.abs(x - y).max() <= 1e-5
    a.close()


@pytest.mark.parametrize("kind", ["pile", "cloth", "mixed", "surface"])
def test_recorded_steps_of_every_material_same_bits(pfsim, monkeypatch, kind):
    """Plain scenes through the step that records their graphs and several
    recorded ones, with a dt that changes every frame: the bits of the same
    scenes stepped without graphs, for contacts, shape matching, a full cloth,
    fluid with soft bodies and a moving collider, and surface effects."""
    from pfsim import _native as N
    from pfsim import recipe as R
    from pfsim import workloads as W

    monkeypatch.setenv("PFSIM_NBR_PATH", "0")  # the autotuner could pick another path for each
    if kind == "pile":
        rec = W.softbody_pile(6000, seed=2, per_body=300)
        rec.loop.contact = True
    elif kind == "cloth":
        rec = W.cloth_sheet(40, seed=3, bend_compliance=1e-5, tethers=True, stretch_tolerance=0.06,
                            wind=(0.8, 0.0, 1.5), damping=0.2)
    elif kind == "mixed":
        rec = W.mixed_scene(6000, 4000, 4, seed=4)
    else:
        rec = W.dam_break(3000, seed=5)
        o = rec.materials[0][1]
        o.surface_tension, o.vorticity = 0.05, 0.02
    a = R.NativeBackend().build(rec)
    b = R.Batch([R.NativeBackend().build(rec)], use_graph=False)
    for k in range(9):
        dt = (1 / 60, 1 / 75, 1 / 50)[k % 3]
        a.step(dt)
        b.step(dt)
        for f in (N.PF_FIELD_POSITIONS, N.PF_FIELD_VELOCITIES):
            assert np.array_equal(a.readback(f), b.readback(0, f)), k
    a.close()
    b.close()


def test_recorded_steps_follow_a_moved_sdf_collider(oracle):
    """An SDF sphere that starts to move once the steps are recorded, under
    particles that rest on it and fall past it: the oracle's positions within
    1e-5 of the metre they stand in, frame by frame."""
    from pfsim import _native as N
    from pfsim import recipe as R

    r = np.random.default_rng(9)
    pos = np.concatenate([r.uniform(-0.2, 0.2, (60, 1)), r.uniform(0.26, 0.6, (60, 1)),
                          r.uniform(-0.2, 0.2, (60, 1))], 1).astype(np.float32)
    rec = R.Recipe(capacity=60, radius=0.01, uploads=[R.Upload(0, pos, None, np.full(60, 100.0, np.float32))],
                   sdfs=[R.sphere_sdf((0.0, 0.0, 0.0), 0.25)], loop=R.LoopOpts(substeps=2, iterations=2))
    a, b = R.NativeBackend().build(rec), oracle.OracleBackend(precision=32).build(rec)
    for k in range(12):
        if k >= 5:
            at, q = (C.c_float * 3)(0.01 * (k - 4), 0.02 * (k - 4), 0.0), (C.c_float * 4)(0.0, 0.0, 0.0, 1.0)
            N.check(N.lib().pf_set_sdf_transform(a.h, 0, at, q, 1.0))
            oracle.check(oracle.lib().or_set_sdf_transform(b.h, 0, at, q, 1.0))
        a.step(1 / 60)
        b.step(1 / 60)
        x, y = a.readback(N.PF_FIELD_POSITIONS), b.readback(N.PF_FIELD_POSITIONS)
        assert np.abs(x - y).max() <= 1e-5, k
    a.close()


def test_threads_read_one_scene_at_once(pfsim):
    """Threads that read different fields of one scene at the same time, one
    of them the whole batch's positions, get what one thread alone reads."""
    from concurrent.futures import ThreadPoolExecutor
    from threading import Barrier

    from pfsim import _native as N
    from pfsim import recipe as R
    from pfsim import workloads as W

    w = R.Batch([R.NativeBackend().build(W.dam_break(30000, seed=51))])
    for _ in range(3):
        w.step(1 / 60)

    def positions():
        out = np.empty((w.capacities[0], 4), np.float32)
        N.check(N.lib().pf_batch_read_positions(w.h, out.ctypes.data_as(C.POINTER(C.c_float)), out.nbytes))
        return out

    fields = [N.PF_FIELD_POSITIONS, N.PF_FIELD_VELOCITIES, N.PF_FIELD_DENSITY, N.PF_FIELD_INV_MASS, N.PF_FIELD_LAMBDA]
    reads = [lambda f=f: w.readback(0, f) for f in fields] + [positions]
    alone = [r() for r in reads]
    start = Barrier(len(reads))

    def reader(k):
        start.wait(60)
        return sum(not np.array_equal(reads[k](), alone[k]) for _ in range(60))

    with ThreadPoolExecutor(len(reads)) as pool:
        assert list(pool.map(reader, range(len(reads)))) == [0] * len(reads)
    w.close()


def test_read_from_a_thread_on_another_device(pfsim):
    """A thread whose current device is not the scene's reads the scene."""
    from concurrent.futures import ThreadPoolExecutor

    import torch

    from pfsim import _native as N
    from pfsim import recipe as R
    from pfsim import workloads as W

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    s = R.NativeBackend().build(W.dam_break(5000, seed=52))
    s.step(1 / 60)
    fields = [N.PF_FIELD_POSITIONS, N.PF_FIELD_DENSITY]

    def elsewhere():
        torch.cuda.set_device(1)
        return [s.readback(f) for f in fields]

    with ThreadPoolExecutor(1) as pool:
        got = pool.submit(elsewhere).result()
    for f, a in zip(fields, got):
        assert np.array_equal(a, s.readback(f))
    s.close()
