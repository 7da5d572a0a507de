"""Barnes-Hut on the GPU against grav_sim.

* Octree (construct_octree): bounding-box width, Morton keys, sorted order,
  node numbering and topology, and internal-node mass / centre of mass are
  bit-exact to the reference (tolerance 0).
* Walk: GRAV_GPU_BARNES_HUT_COMPAT (113) reproduces the reference's walk,
  including its zero-mass leaves and its key indexing, and
  GRAV_GPU_BARNES_HUT (103) the corrected walk of the oracle.  Every
  opening decision equals the oracle's (the GPU's interaction counts are
  identical), and accelerations, made of FP32 terms, are held to:
  |a_i - a_ref,i| <= 1e-5 * A_i with A_i the sum of the magnitudes of
  particle i's terms, and per-particle relative error median <= 1e-6,
  99th percentile <= 1e-5.
"""
import ctypes

import numpy as np
import pytest

from conftest import cases, golden

pytestmark = pytest.mark.gpu

TREE_KEYS = ("keys", "sorted_indices", "num_particles", "num_children", "first_particle")


def gpu_octree(lib, g, x, m, leaf, method=3):
    system, keep = g.make_system(x, m, 1.0)
    t = g.LinearOctree()
    p = g.AccelerationParam(method, 1.0, 0.0, int(leaf))
    st = lib.construct_octree(ctypes.byref(t), ctypes.byref(system), ctypes.byref(p), None, -1.0)
    assert st.return_code == 0, g.take_traceback(lib, st)
    n, nn = system.num_particles, t.num_internal_nodes
    out = dict(
        box_width=t.box_width, num_nodes=nn,
        keys=np.ctypeslib.as_array(t.particle_morton_indices_deepest_level, (n,)).copy(),
        sorted_indices=np.ctypeslib.as_array(t.sorted_indices, (n,)).copy(),
        num_particles=np.ctypeslib.as_array(t.tree_num_particles, (nn,)).copy(),
        num_children=np.ctypeslib.as_array(t.tree_num_internal_children, (nn,)).copy(),
        first_particle=np.ctypeslib.as_array(t.tree_first_particle_sorted_idx, (nn,)).copy(),
        first_child=np.ctypeslib.as_array(t.tree_first_internal_children_idx, (nn,)).copy(),
        mass=np.ctypeslib.as_array(t.tree_mass, (nn,)).copy(),
        com=np.stack([np.ctypeslib.as_array(t.tree_center_of_mass_x, (nn,)).copy(),
                      np.ctypeslib.as_array(t.tree_center_of_mass_y, (nn,)).copy(),
                      np.ctypeslib.as_array(t.tree_center_of_mass_z, (nn,)).copy()], 1),
    )
    lib.free_linear_octree(ctypes.byref(t))
    del keep
    return out


def assert_same_tree(gt, ref, name=""):
    assert gt["num_nodes"] == len(ref["num_particles"]), name
    assert gt["box_width"] == float(ref["box_width"]), name
    for k in TREE_KEYS:
        assert np.array_equal(gt[k], ref[k]), (name, k)
    internal = ref["num_children"] > 0
    assert np.array_equal(gt["first_child"][internal], ref["first_child"][internal]), name
    assert np.array_equal(gt["mass"][internal], ref["mass"][internal]), name
    assert np.array_equal(gt["com"][internal], ref["com"][internal]), name


def test_octree_bitexact_golden(lib, g):
    for name, c in cases(golden("octree")).items():
        gt = gpu_octree(lib, g, c["x"], c["m"], int(c["leaf"]))
        assert_same_tree(gt, c, name)


@pytest.mark.parametrize("n,leaf", [(1, 1), (2, 1), (9, 2), (5000, 1), (5000, 3), (100000, 1),
                                    (100000, 16)])
def test_octree_bitexact_fresh(lib, g, orc, wl, n, leaf):
    x, v, m = wl.plummer(n, 1000 + n + leaf)
    gt = gpu_octree(lib, g, x, m, leaf)
    ref = orc.build_tree(x, m, leaf, True)
    assert_same_tree(gt, ref)
    # the corrected tree gives leaves their own mass and centre of mass
    gf = gpu_octree(lib, g, x, m, leaf, method=g.METHOD_GPU_BARNES_HUT)
    rf = orc.build_tree(x, m, leaf, False)
    assert np.array_equal(gf["mass"], rf["mass"]) and np.array_equal(gf["com"], rf["com"])


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4097])
@pytest.mark.parametrize("leaf", [1, 6, 5000])
def test_octree_bitexact_at_scan_tile_edges(lib, g, orc, wl, n, leaf):
    """Particle counts next to the 2,048-particle tile of the topology scans (leaf 6: internal
    nodes on both sides of its 256-node tile; leaf 5000: the root's children are all leaves), with
    coincident particles, whose chains of nodes reach depth 21, on both sides of a tile's end."""
    x, v, m = wl.plummer(n, n + leaf)
    order = np.argsort(orc.morton(x, *orc.bbox(x)), kind="stable")
    x[order[2040:2046]] = x[order[2040]]
    gt = gpu_octree(lib, g, x, m, leaf)
    assert_same_tree(gt, orc.build_tree(x, m, leaf, True))


@pytest.mark.parametrize("leaf", [2, 7, 8, 9, 16, 33])
def test_octree_bitexact_at_run_edges(lib, g, orc, wl, leaf):
    """The climb adds the particles of consecutive leaf children eight at a time."""
    x, v, m = wl.galaxy_pair(6000, 40 + leaf)
    assert_same_tree(gpu_octree(lib, g, x, m, leaf), orc.build_tree(x, m, leaf, True))


@pytest.mark.parametrize("n", [1023, 1024, 1025, 200000, 200001, 400000, 400001])
def test_octree_bitexact_at_sort_tile_edges(lib, g, orc, wl, n):
    """Sort tiles of 1,024, 2,048 (above 200,000 particles) and 4,096 (above 400,000)."""
    x, v, m = wl.galaxy_pair(n, 3)
    assert_same_tree(gpu_octree(lib, g, x, m, 16), orc.build_tree(x, m, 16, True))


def test_octree_bitexact_galaxy_collision_2097152(lib, g, orc, wl):
    """Morton keys, order and tree of the galaxy-collision workload at full
    size, bit-exact."""
    x, v, m = wl.galaxy_pair(2097152, 4)
    gt = gpu_octree(lib, g, x, m, 1)
    ref = orc.build_tree(x, m, 1, True)
    assert_same_tree(gt, ref)


def check_terms(a, ref, absum):
    diff = np.linalg.norm(a - ref, axis=1)
    assert np.all(diff <= 1e-5 * absum + 1e-300), float(np.max(diff / (absum + 1e-300)))
    mag = np.linalg.norm(ref, axis=1)
    nz = mag > 0
    rel = diff[nz] / mag[nz]
    med, p99 = float(np.median(rel)), float(np.quantile(rel, 0.99))
    assert med <= 1e-6 and p99 <= 1e-5, (med, p99)
    return med, p99


def gpu_counts(lib):
    c = (ctypes.c_longlong * 2)()
    assert lib.gsgpu_last_interaction_counts(c) == 0
    return int(c[0]), int(c[1])


def test_compat_walk_golden(lib, g, orc):
    for name, c in cases(golden("barnes_hut")).items():
        leaf = int(c["leaf"])
        for th in (0.5, 1.0):
            a = g.acceleration(lib, c["x"], c["m"], 1.0, g.METHOD_GPU_BARNES_HUT_COMPAT,
                               opening_angle=th, softening_length=0.01,
                               max_num_particles_per_leaf=leaf)
            a_o, cnt, mag = orc.bh_counts(c["x"], c["m"], 1.0, 0.01, th, leaf, True)
            assert np.array_equal(a_o, c[f"a_theta{th}"])
            assert gpu_counts(lib) == (int(cnt[:, 0].sum()), int(cnt[:, 1].sum())), (name, th)
            check_terms(a, c[f"a_theta{th}"], mag)


@pytest.mark.parametrize("compat", [True, False])
@pytest.mark.parametrize("theta,leaf", [(0.5, 1), (1.0, 1), (0.7, 8)])
def test_walk_vs_oracle(lib, g, orc, wl, compat, theta, leaf):
    x, v, m = wl.galaxy_pair(65536, 11)
    method = g.METHOD_GPU_BARNES_HUT_COMPAT if compat else g.METHOD_GPU_BARNES_HUT
    a = g.acceleration(lib, x, m, 1.0, method, opening_angle=theta, softening_length=0.01,
                       max_num_particles_per_leaf=leaf)
    a_o, cnt, mag = orc.bh_counts(x, m, 1.0, 0.01, theta, leaf, compat)
    assert gpu_counts(lib) == (int(cnt[:, 0].sum()), int(cnt[:, 1].sum()))
    check_terms(a, a_o, mag)


@pytest.mark.parametrize("compat", [True, False])
@pytest.mark.parametrize("n,theta,leaf", [(2, 0.5, 1), (31, 0.5, 1), (32, 0.5, 1), (33, 0.9, 2),
                                          (65, 0.8, 3), (1000, 0.5, 40), (4097, 0.3, 1),
                                          (62208, 0.7, 1), (62240, 0.7, 1)])
def test_walk_edges_vs_oracle(lib, g, orc, wl, compat, n, theta, leaf):
    """Warps that are not full, leaves longer than a warp, lists around their capacity, and both
    forms of the walk (62,208 particles are 1,944 warps, the last count that a block each walks).
    Every decision equals the oracle's."""
    x, v, m = wl.plummer(n, n)
    if n > 100:
        x[60:64] = x[70]   # coincident particles
    method = g.METHOD_GPU_BARNES_HUT_COMPAT if compat else g.METHOD_GPU_BARNES_HUT
    a = g.acceleration(lib, x, m, 1.0, method, opening_angle=theta, softening_length=0.01,
                       max_num_particles_per_leaf=leaf)
    a_o, cnt, mag = orc.bh_counts(x, m, 1.0, 0.01, theta, leaf, compat)
    assert gpu_counts(lib) == (int(cnt[:, 0].sum()), int(cnt[:, 1].sum()))
    check_terms(a, a_o, mag)


def test_reference_entry_point_acceleration_barnes_hut(lib, g, orc, wl):
    """acceleration_barnes_hut() with the reference's method code 3 runs the
    reference-compatible GPU walk."""
    x, v, m = wl.plummer(3000, 3)
    system, keep = g.make_system(x, m, 1.0)
    a = np.empty((3000, 3))
    p = g.AccelerationParam(3, 0.5, 0.01, 1)
    lib.acceleration_barnes_hut.restype = g.ErrorStatus
    st = lib.acceleration_barnes_hut(a.ctypes.data_as(g.c_double_p), ctypes.byref(system),
                                     ctypes.byref(p))
    assert st.return_code == 0
    a_o, cnt, mag = orc.bh_counts(x, m, 1.0, 0.01, 0.5, 1, True)
    check_terms(a, a_o, mag)


@pytest.mark.parametrize("theta", [0.5, 1.0])
def test_quadrupole_walk_vs_oracle(lib, g, orc, wl, theta):
    """GRAV_GPU_BARNES_HUT_QUAD: same opening decisions as the corrected walk,
    cells add monopole + quadrupole terms; quadrupoles composed bottom-up on
    the GPU (parallel-axis shifts) against the oracle's direct per-node sums."""
    x, v, m = wl.galaxy_pair(32768, 12)
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_QUAD, opening_angle=theta,
                       softening_length=0.01, max_num_particles_per_leaf=1)
    a_o, mag, q = orc.bh_quad(x, m, 1.0, 0.01, theta, 1)
    _, cnt, _ = orc.bh_counts(x, m, 1.0, 0.01, theta, 1, False)
    assert gpu_counts(lib) == (int(cnt[:, 0].sum()), int(cnt[:, 1].sum()))
    check_terms(a, a_o, mag)


def test_fixed_walk_accuracy_vs_direct_sum(lib, g, orc, wl):
    """Corrected multipoles: theta=0.5 reaches ~1e-3 median error against the
    FP64 direct sum on the galaxy model (the reference's walk does not)."""
    x, v, m = wl.galaxy_pair(131072, 5)
    rows = np.random.default_rng(1).choice(x.shape[0], 2048, replace=False).astype(np.int32)
    exact = orc.direct_rows(x, m, 1.0, 0.01, rows)
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT, opening_angle=0.5,
                       softening_length=0.01, max_num_particles_per_leaf=1)
    err = orc.rel_err(a[rows], exact)
    print(f"fixed theta=0.5 median {np.median(err):.3g} p99 {np.quantile(err, 0.99):.3g}")
    assert np.median(err) < 3e-3


@pytest.mark.parametrize("theta,leaf", [(0.5, 1), (0.8, 1), (0.5, 64)])
def test_group_walk_accuracy(lib, g, orc, wl, theta, leaf):
    """Group walk (106): its group opening criterion implies the per-particle
    one for every particle, so it is at least about as accurate as the
    per-particle quadrupole walk (105) at the same theta.  leaf=64 exercises
    leaves that overflow one list round."""
    x, v, m = wl.galaxy_pair(131072, 7)
    rows = np.random.default_rng(3).choice(x.shape[0], 2048, replace=False).astype(np.int32)
    exact = orc.direct_rows(x, m, 1.0, 0.01, rows)
    kw = dict(opening_angle=theta, softening_length=0.01, max_num_particles_per_leaf=leaf)
    a_g = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, **kw)
    cells, pairs = gpu_counts(lib)
    a_q = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_QUAD, **kw)
    e_g = np.median(orc.rel_err(a_g[rows], exact))
    e_q = np.median(orc.rel_err(a_q[rows], exact))
    print(f"theta={theta} leaf={leaf}: group {e_g:.3g} ({cells} cells, {pairs} pairs), "
          f"per-particle quad {e_q:.3g}")
    assert np.isfinite(a_g).all()
    assert e_g <= 1.1 * e_q
    assert cells > 0 and pairs > 0


def group_origins(orc, x, m, leaf=16, size=32):
    """First particle of the group that each particle is walked with: runs of
    consecutive children of at most `size` particles in a larger cell, cut into
    pieces of `size`; a piece that does not fit its cell (it holds a particle at
    the box maximum, whose key wraps) is walked particle by particle."""
    t = orc.build_tree(x, m, leaf, False)
    num, kids, p0, c0 = (np.asarray(t[k]) for k in ("num_particles", "num_children",
                                                    "first_particle", "first_child"))
    ids = np.asarray(t["sorted_indices"])
    first = np.empty(len(x), int)

    def cut(begin, count, cell):
        for b in range(begin, begin + count, size):
            own = ids[b:min(b + size, begin + count)]
            fits = np.ptp(x[own], axis=0).max() <= t["box_width"] / 2.0 ** t["depth"][cell]
            first[own] = own[0] if fits else own

    if num[0] <= size or kids[0] == 0:
        cut(0, len(x), 0)
    for q in np.where((num > size) & (kids > 0))[0]:
        begin = p0[q]
        for c in range(c0[q], c0[q] + kids[q]):
            if num[c] > size:
                cut(begin, p0[c] - begin, q)
                begin = p0[c] + num[c]
                if kids[c] == 0:
                    cut(p0[c], num[c], c)
        cut(begin, p0[q] + num[q] - begin, q)
    return first


def fp32_offsets(x, origin):
    """Positions as the walk forms them: FP32 offsets from a group's first
    particle, from double-float copies about the frame's centre."""
    c = x - 0.5 * (x.min(0) + x.max(0))
    hi = c.astype(np.float32)
    lo = (c - hi).astype(np.float32)
    return ((hi - hi[origin]) + (lo - lo[origin])).astype(np.float64)


@pytest.mark.parametrize("clusters,size,eps", [
    (1, 1, 0.0), (1, 2, 0.0), (1, 16, 0.0), (1, 17, 0.0), (2, 33, 0.0), (3, 15, 0.0), (4, 32, 1e-4),
    (5, 31, 0.0), (31, 16, 0.0), (129, 17, 0.0), (130, 1, 0.0), (131, 33, 1e-4), (257, 20, 0.0),
    (4096, 33, 0.0), (4096, 33, 1e-4)])
def test_group_walk_lists_vs_direct_sum(lib, g, orc, clusters, size, eps):
    """Group walk against the FP64 direct sum of the positions it forms (FP32
    offsets from the group's first particle), where both are the same: compact
    clusters on a jittered grid and an angle at which an accepted cell holds one
    cluster.  Group sizes around one row (16) and a full group (32), cell lists
    around whole turns and around the list's capacity (128), and both forms of
    the walk (a CTA per group; 4,096 clusters of 33 make enough groups for a warp
    each).  Cell side < theta d <= 0.43 h, so its diagonal is below the clusters'
    separation 0.8 h; a cluster's radius is 0.005 h, so beyond the quadrupole a
    cell's term is off by at most 4 (0.01 / 0.8)^3 = 8e-6 of itself, and the FP32
    terms add less than 4e-6 of the sum of magnitudes."""
    rng = np.random.default_rng(clusters * 64 + size)
    grid = int(np.ceil(clusters ** (1.0 / 3.0) - 1e-9))
    h = 1.0 / grid
    k = np.arange(clusters)
    c = np.stack([k % grid, k // grid % grid, k // grid // grid], 1) * h
    c = c + rng.uniform(-0.1 * h, 0.1 * h, c.shape)
    d = rng.normal(size=(clusters, size, 3))
    d *= (0.005 * h * rng.uniform(0.2, 1.0, (clusters, size, 1))) / np.linalg.norm(d, axis=2, keepdims=True)
    x = np.ascontiguousarray((c[:, None, :] + d).reshape(-1, 3))
    n = len(x)
    m = rng.uniform(0.5, 1.5, n) / n
    rows = rng.permutation(n)[:256].astype(np.int32)
    # a particle on the box maximum sits in a cell on the far side (its key
    # wraps), whose centre is not near its cluster: those clusters are left out
    plain = ~np.isin(rows // size, x.argmax(0) // size)
    rows = rows[plain] if plain.any() else rows
    first = group_origins(orc, x, m)
    exact, absum = np.empty((len(rows), 3)), np.empty((len(rows), 1))
    for i, r in enumerate(rows):
        off = fp32_offsets(x, first[r])
        d = off - off[r]
        r2 = (d * d).sum(1)
        w = m / np.where(r2 > 0.0, (r2 + eps * eps) ** 1.5, 1.0)
        exact[i] = (w[:, None] * d).sum(0)
        absum[i] = (w * np.sqrt(r2)).sum()
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, opening_angle=0.25 / grid,
                       softening_length=eps)
    assert np.isfinite(a).all()
    assert (np.abs(a[rows] - exact) <= 1.2e-5 * absum).all()


def test_group_walk_degenerate_and_unsoftened(lib, g, orc, wl):
    """A 200-particle coincident cluster (one depth-21 leaf with more
    particles than one list round) with softening, and an unsoftened
    Plummer sphere (the particle's own term is skipped)."""
    x, v, m = wl.plummer(20000, 11)
    x[100:300] = x[50]
    rows = np.arange(40, 340, dtype=np.int32)
    exact = orc.direct_rows(x, m, 1.0, 0.01, rows)
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, opening_angle=0.6,
                       softening_length=0.01, max_num_particles_per_leaf=1)
    assert np.isfinite(a).all()
    assert np.median(orc.rel_err(a[rows], exact)) < 2e-3
    x2, v2, m2 = wl.plummer(20000, 12)
    rows2 = np.random.default_rng(4).choice(20000, 512, replace=False).astype(np.int32)
    exact2 = orc.direct_rows(x2, m2, 1.0, 0.0, rows2)
    a2 = g.acceleration(lib, x2, m2, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, opening_angle=0.5,
                        softening_length=0.0, max_num_particles_per_leaf=1)
    assert np.isfinite(a2).all()
    assert np.median(orc.rel_err(a2[rows2], exact2)) < 2e-3


@pytest.mark.parametrize("method", [3, 13, 5, 6])
def test_node_capacity_overflow(lib, g, orc, wl, method):
    """2,048 coincident pairs with one particle per leaf: each pair splits
    down to the depth limit, 36,951 nodes (the oracle's count) against a
    capacity of 4N + 4096 = 20,480.  The build stops at the capacity, the
    kernels after it do no work, and the call reports GRAV_MEMORY_ERROR;
    the same engine then serves a normal input."""
    rng = np.random.default_rng(6)
    x = np.repeat(rng.random((2048, 3)), 2, axis=0)
    m = np.full(4096, 1.0 / 4096)
    assert orc.build_tree(x, m, 1, False)["num_nodes"] > 4 * 4096 + 4096
    gpu = method + 100
    with pytest.raises(g.GravError) as e:
        g.acceleration(lib, x, m, 1.0, gpu, opening_angle=0.5, softening_length=0.01,
                       max_num_particles_per_leaf=1)
    assert e.value.code == g.GRAV_MEMORY_ERROR
    if method == 3:
        system, keep = g.make_system(x, m, 1.0)
        t = g.LinearOctree()
        p = g.AccelerationParam(3, 1.0, 0.0, 1)
        st = lib.construct_octree(ctypes.byref(t), ctypes.byref(system), ctypes.byref(p),
                                  None, -1.0)
        assert st.return_code == g.GRAV_MEMORY_ERROR
        g.take_traceback(lib, st)
    x2, _, m2 = wl.plummer(4096, 3)
    a = g.acceleration(lib, x2, m2, 1.0, gpu, opening_angle=0.5, softening_length=0.01,
                       max_num_particles_per_leaf=1)
    assert np.isfinite(a).all()
    if method in (3, 13):   # the oracle's walk, term for term
        a_o, cnt, mag = orc.bh_counts(x2, m2, 1.0, 0.01, 0.5, 1, method == 13)
        check_terms(a, a_o, mag)
    else:
        rows = np.arange(0, 4096, 16, dtype=np.int32)
        err = orc.rel_err(a[rows], orc.direct_rows(x2, m2, 1.0, 0.01, rows))
        assert np.median(err) < 5e-3


def test_group_walk_in_simulation(lib, g, wl):
    """The group walk drives launch_simulation (graph-captured leapfrog)."""
    x, v, m = wl.galaxy_pair(32768, 8)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=4, dt=1e-3,
                                       tf=0.01, method=g.METHOD_GPU_BARNES_HUT_GROUP,
                                       opening_angle=0.5, softening_length=0.01,
                                       max_num_particles_per_leaf=1)
    assert np.isfinite(xo).all() and np.isfinite(vo).all()
    assert np.abs(xo - x).max() < 0.1


def test_group_walk_galaxy_1m(lib, g, orc, wl):
    """The full-size galaxy model: dense centres stress the traversal stack
    (an overflow would be reported as an error), accuracy stays below the
    per-particle criterion's."""
    x, v, m = wl.galaxy_pair(1048576, 5)
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, opening_angle=0.5,
                       softening_length=0.01, max_num_particles_per_leaf=1)
    rows = np.random.default_rng(5).choice(x.shape[0], 256, replace=False).astype(np.int32)
    err = orc.rel_err(a[rows], orc.direct_rows(x, m, 1.0, 0.01, rows))
    print(f"group walk N=1048576 theta=0.5: median {np.median(err):.3g}")
    assert np.isfinite(a).all() and np.median(err) < 1e-3


def test_group_walk_particles_on_box_maximum(lib, g, orc, wl):
    """Particles exactly on the bounding-box maximum get Morton coordinate 0
    (the reference's wrap) and sit in a cell on the far side: their group
    does not fit its cell and is walked particle by particle, with the same
    accuracy as everyone else."""
    x, v, m = wl.plummer(50000, 13)
    hi = x.max(axis=0)
    x[7] = hi
    x[8] = hi - 1e-9
    x[9, 0] = hi[0]
    rows = np.array([7, 8, 9, 10, 11], dtype=np.int32)
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, opening_angle=0.5,
                       softening_length=0.01, max_num_particles_per_leaf=1)
    err = orc.rel_err(a[rows], orc.direct_rows(x, m, 1.0, 0.01, rows))
    assert np.isfinite(a).all() and err.max() < 5e-3


def test_group_walk_monopole_vs_per_particle(lib, g, orc, wl):
    """Monopole group walk (107): at least about as accurate as the
    per-particle monopole walk (103) at the same theta."""
    x, v, m = wl.galaxy_pair(131072, 9)
    rows = np.random.default_rng(6).choice(x.shape[0], 2048, replace=False).astype(np.int32)
    exact = orc.direct_rows(x, m, 1.0, 0.01, rows)
    kw = dict(opening_angle=0.5, softening_length=0.01, max_num_particles_per_leaf=1)
    e_g = np.median(orc.rel_err(g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP_MONO,
                                               **kw)[rows], exact))
    e_p = np.median(orc.rel_err(g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT, **kw)[rows],
                                exact))
    print(f"monopole: group {e_g:.3g}, per-particle {e_p:.3g}")
    assert e_g <= 1.1 * e_p


def test_width_division_matches_ddiv(lib):
    """The Morton keys' division-free quotients by the box width equal
    __ddiv_rn bit for bit: 2^26 samples of widths in [2^-100, 2^100] and
    dividends of every class and next to rounding ties."""
    import ctypes
    lib.gsgpu_width_division_selftest.restype = ctypes.c_int
    lib.gsgpu_width_division_selftest.argtypes = [ctypes.c_longlong, ctypes.c_ulonglong,
                                                  ctypes.POINTER(ctypes.c_longlong)]
    bad = ctypes.c_longlong(-1)
    for seed in (1, 2):
        assert lib.gsgpu_width_division_selftest(1 << 26, seed, ctypes.byref(bad)) == 0
        assert bad.value == 0


@pytest.mark.parametrize("method", [103, 105])
@pytest.mark.parametrize("case", ["pair", 1e-7, 1.0, 1e6, 1e8])
def test_walk_at_close_pairs_and_scales(lib, g, orc, wl, method, case):
    """Distances far from one, unsoftened: two particles 1e-7 apart among 1,000 others, and a
    galaxy pair scaled as a whole.  No power of the distance in a term may leave the FP32 range
    before m / r^3 does; the bounds are those of the walk at any scale."""
    if case == "pair":
        x, v, m = wl.plummer(1002, 6)
        x[501] = x[500] + np.array([6e-8, -8e-8, 0.0])
    else:
        x, v, m = wl.galaxy_pair(4096, 17)
        x = x * case
    a = g.acceleration(lib, x, m, 1.0, method, opening_angle=0.5, softening_length=0.0,
                       max_num_particles_per_leaf=1)
    assert np.isfinite(a).all()
    if method == 105:
        a_o, mag, _ = orc.bh_quad(x, m, 1.0, 0.0, 0.5, 1)
    else:
        a_o, _, mag = orc.bh_counts(x, m, 1.0, 0.0, 0.5, 1, False)
    check_terms(a, a_o, mag)


@pytest.mark.parametrize("log2_scale", [-10, 23, 27])
def test_group_walk_scales(lib, g, wl, log2_scale):
    """Scaling every position by a power of two scales each FP32 operation of the walk exactly
    while nothing leaves the range, so the accelerations scale by its inverse square.  (r^-7,
    once a factor of the quadrupole term, leaves it at each of these scales; below 2^-100 of
    the largest the terms are subnormal and round differently: 1e-6.)"""
    x, v, m = wl.galaxy_pair(20000, 23)
    kw = dict(opening_angle=0.5, softening_length=0.0, max_num_particles_per_leaf=1)
    scale = 2.0 ** log2_scale
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, **kw)
    b = g.acceleration(lib, x * scale, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, **kw) * scale ** 2
    assert np.isfinite(b).all()
    assert (np.linalg.norm(a - b, axis=1) <= 1e-6 * np.linalg.norm(a, axis=1)).all()


@pytest.mark.parametrize("method,what", [(113, "position"), (103, "mass"), (105, "mass")])
def test_walk_with_a_particle_that_is_not_finite(lib, g, orc, wl, method, what):
    """A particle that is not finite reaches those that its leaf is opened for, and no others of
    their warps: with the reference's walk (113), where far leaves weigh nothing, the rest stay
    finite, and the particle with an infinite mass itself feels the others alone."""
    x, v, m = wl.galaxy_pair(3000, 19)
    k = 1234
    if what == "position":
        x[k, 1] = np.nan
    else:
        m[k] = np.inf
    a = g.acceleration(lib, x, m, 1.0, method, opening_angle=0.5, softening_length=0.01,
                       max_num_particles_per_leaf=1)
    a_o, _, mag = orc.bh_counts(x, m, 1.0, 0.01, 0.5, 1, method == 113)
    finite = np.isfinite(a_o).all(axis=1)
    assert finite.any() and not finite.all() and (what == "position" or finite[k])
    assert np.array_equal(np.isfinite(a).all(axis=1), finite)
    if method != 105:
        check_terms(a[finite], a_o[finite], mag[finite])


@pytest.mark.parametrize("method,what", [(103, "mass"), (105, "mass"), (105, "quadrupole")])
def test_walk_with_cells_beyond_fp32(lib, g, orc, method, what):
    """A cell whose mass or quadrupole is infinite in FP32 reaches the particles that accept it,
    and not those of their warps that open it; which ones follows from the oracle's tree.  Among
    light particles a tight clump of 64 masses of 1e37, or a pair of 1e34 a thousand apart, whose
    other terms stay in range."""
    rng = np.random.default_rng(8)
    n, theta = 500, 0.7
    scale, k, heavy = (100.0, 64, 1e37) if what == "mass" else (1e5, 2, 1e34)
    x = rng.uniform(-scale, scale, (n, 3))
    x[:k] = 0.4 * scale
    x[:k] += rng.uniform(-0.002, 0.002, (k, 3)) if what == "mass" else [[-500.0] * 3, [500.0] * 3]
    x[k:k + 64] = 0.4 * scale + rng.uniform(-0.09 * scale, 0.09 * scale, (64, 3))
    m = np.ones(n)
    m[:k] = heavy
    t = orc.build_tree(x, m, 1, False)
    q = orc.bh_quad(x, m, 1.0, 0.0, theta, 1)[2]
    first, num, side = t["first_particle"], t["num_particles"], t["box_width"] / 2.0 ** t["depth"]
    big = t["mass"] if what == "mass" else np.abs(q).max(axis=1)
    big = big > 3.4028236e38
    place = np.empty(n, int)
    place[t["sorted_indices"]] = np.arange(n)
    expect = np.zeros(n, bool)
    for i in range(n):
        stack = [0]
        while stack:
            c = stack.pop()
            inside = first[c] <= place[i] < first[c] + num[c]
            if c and not inside and side[c] ** 2 < theta ** 2 * ((t["com"][c] - x[i]) ** 2).sum():
                expect[i] |= big[c]
            elif t["num_children"][c]:
                stack += range(t["first_child"][c], t["first_child"][c] + t["num_children"][c])
    assert 20 < expect.sum() < n - 20
    a = g.acceleration(lib, x, m, 1.0, method, opening_angle=theta,
                       softening_length=1.0 if what == "mass" else 0.0,
                       max_num_particles_per_leaf=1)
    assert np.array_equal(~np.isfinite(a).all(axis=1), expect)


@pytest.mark.parametrize("n", [400, 20000])
def test_quadrupole_walks_with_massless_particles(lib, g, orc, wl, n):
    """Massless particles (cells of them have no centre of mass) add nothing to the quadrupoles
    of the cells above: 105 against the oracle, whose quadrupoles are sums over a node's
    particles, and 106 at least about as accurate."""
    x, v, m = wl.galaxy_pair(n, 29)
    m = np.where(np.random.default_rng(1).random(n) < 0.7, 0.0, m)
    kw = dict(opening_angle=0.5, softening_length=0.01, max_num_particles_per_leaf=1)
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_QUAD, **kw)
    b = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_GROUP, **kw)
    assert np.isfinite(a).all() and np.isfinite(b).all()
    a_o, mag, _ = orc.bh_quad(x, m, 1.0, 0.01, 0.5, 1)
    check_terms(a, a_o, mag)
    rows = np.arange(0, n, max(1, n // 400), dtype=np.int32)
    exact = orc.direct_rows(x, m, 1.0, 0.01, rows)
    assert np.median(orc.rel_err(b[rows], exact)) <= 1.1 * np.median(orc.rel_err(a[rows], exact))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("theta", [0.5, 1.5, 5.0])
def test_compat_walk_with_a_lost_coordinate(lib, g, orc, axis, theta):
    """One coordinate of one particle is NaN, and of the centres of the cells it is in: no
    particle accepts those, however far away they are in the other coordinates."""
    rng = np.random.default_rng(12)
    x = rng.integers(-4, 5, (1500, 3)).astype(float) + rng.uniform(-0.2, 0.2, (1500, 3))
    m = np.ones(len(x))
    x[777, axis] = np.nan
    a = g.acceleration(lib, x, m, 1.0, g.METHOD_GPU_BARNES_HUT_COMPAT, opening_angle=theta,
                       softening_length=0.05, max_num_particles_per_leaf=1)
    a_o, _, mag = orc.bh_counts(x, m, 1.0, 0.05, theta, 1, True)
    finite = np.isfinite(a_o).all(axis=1)
    assert finite.any() and not finite.all()
    assert np.array_equal(np.isfinite(a).all(axis=1), finite)
    check_terms(a[finite], a_o[finite], mag[finite])
