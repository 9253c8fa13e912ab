"""GPU tests of the TreePM walk's group sizes, pair polynomials and periodic images.

The walk groups neighbouring targets (1, 4, 8 or 16 by their number and density)
and evaluates the pair factor by a polynomial whose degree depends on
r_cut / r_s (a closed form beyond). Every case here opens every node
(theta = 1e-6), so the result is direct summation: the oracle's long-double sum,
to 1e-12 relative RMS in binary64 (700 pairs of a few ulp each) and 1e-5 in the
FP32 form. With theta = 0.5 the same targets give the same accepted set whatever
the group, so the results agree to summation order (1e-12, and 1e-6 in FP32).
"""
import ctypes
import math

import numpy as np
import pytest

import hyowon_b200 as hb
from hyowon_b200 import _native as nat
from hyowon_b200.treepm import short_range_forces

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32": 1e-5}    # against direct summation
SAME = {"fp64": 1e-12, "fp32": 1e-6}   # one group against another


def rel_rms(got, ref):
    g, r = np.stack(got), np.stack(ref)
    return float(np.sqrt(np.sum((g - r) ** 2) / np.sum(r ** 2)))


def points(n, L, seed):
    """Half uniform, half in tight clumps, some across the box edge."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(0, L, (3, n))
    k = n // 2
    centre = rng.uniform(-0.02 * L, L, (3, max(1, n // 300)))
    p[:, :k] = centre[:, rng.integers(0, centre.shape[1], k)] + rng.normal(0, 0.01 * L, (3, k))
    return np.mod(p, L)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ratio", [2.0, 4.5, 5.6, 6.4, 7.5, 12.0])
def test_pair_factor_over_cutoff_ratios(oracle, precision, ratio):
    """Each polynomial degree and the closed form, against the long-double sum."""
    L, n = 24.0, 3000
    x, y, z = points(n, L, 3)
    r_cut, eps = 5.0, 0.04
    t = np.arange(0, n, 7, dtype=np.uint32)
    ref = oracle.short_range_direct(L, x, y, z, 1.5, t, r_cut / ratio, r_cut, eps)
    got = short_range_forces(L, x, y, z, 1.5, t, r_cut / ratio, r_cut, eps, 1e-6, precision)
    assert rel_rms(got[:3], ref) <= TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ratio", [2.0, 3.6, 4.5, 5.4, 6.0, 7.0, 7.5, 8.5])
def test_isolated_pairs_over_the_cutoff_sphere(oracle, precision, ratio):
    """512 pairs with no other source within reach, their separations spread over the
    cutoff sphere up to 0.9999 r_cut: each force is one pair factor. Bound, relative to
    (M_S + |softening term|) / r^3, which the factor equals except where the two cancel
    (r near 7 r_s): binary64, the factor's own nine roundings, its powers and products
    (4e-15 in all) and the rounding of r^2 (up to 6 half ulps) times its logarithmic
    slope, at most 1.5 + q^2 / 4; precision form, 1e-7, the FP32 half ulp and a half."""
    r_cut, side = 1.0, 8
    r_s, cell = r_cut / ratio, 3.2 * r_cut
    eps, L = r_s / 37.0, side * cell
    rng = np.random.default_rng(int(10 * ratio))
    n = side ** 3
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij")).reshape(3, n)
    first = (grid + 0.5) * cell + rng.uniform(-0.05, 0.05, (3, n))
    way = rng.normal(size=(3, n))
    r = r_cut * np.concatenate([np.linspace(0.01, 0.9, n // 2), np.linspace(0.9, 0.9999, n - n // 2)])
    second = first + way / np.linalg.norm(way, axis=0) * r
    x, y, z = (np.concatenate([a, b]) for a, b in zip(first, second))
    every = np.arange(2 * n, dtype=np.uint32)
    args = (r_s, r_cut, eps)
    ref = np.stack(oracle.short_range_direct(L, x, y, z, 1.0, every, *args))
    got = np.stack(short_range_forces(L, x, y, z, 1.0, every, *args, 1e-6, precision)[:3])
    q = np.tile(r, 2) / r_s
    ms = np.array([math.erfc(0.5 * v) for v in q]) + q / math.sqrt(math.pi) * np.exp(-0.25 * q * q)
    soft = np.expm1(-1.5 * np.log1p((eps / r_s / q) ** 2))
    scale = np.linalg.norm(ref, axis=0) * (ms - soft) / np.abs(ms + soft)
    err = np.linalg.norm(got - ref, axis=0) / scale
    bound = (1.5 + 0.25 * q * q) * 6.7e-16 + 4e-15 if precision == "fp64" else 1e-7
    assert np.all(err <= bound), (float(np.max(err)), float(np.max(err / bound)))


@pytest.mark.parametrize("n,nt", [(2, 1), (2, 2), (3, 3), (5, 5), (17, 17), (33, 31), (4097, 4097),
                                  (4097, 2000), (4097, 511), (120011, 120011), (120011, 70000)])
def test_groups_are_direct_summation(oracle, n, nt):
    """Remainders of every group size, and targets denser and sparser than it."""
    L = 30.0
    x, y, z = points(n, L, n)
    rng = np.random.default_rng(n + nt)
    t = rng.permutation(n)[:nt].astype(np.uint32)
    check = np.arange(nt) if nt <= 4097 else rng.choice(nt, 500, replace=False)
    r_cut = 14.0 if n <= 33 else 3.0
    ref = oracle.short_range_direct(L, x, y, z, 1.0, t[check], r_cut / 4.5, r_cut, 0.03)
    got = short_range_forces(L, x, y, z, 1.0, t, r_cut / 4.5, r_cut, 0.03, 1e-6)
    got = [g[check] for g in got[:3]]
    scale = max(float(np.max(np.abs(r))) for r in ref)
    if scale == 0.0:     # no pair within the cutoff
        assert max(float(np.max(np.abs(g))) for g in got) == 0.0
    else:
        assert rel_rms(got, ref) <= TOL["fp64"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("theta", [0.3, 0.5, 0.9, 1.6])
@pytest.mark.parametrize("n,L,r_cut", [(900, 10.0, 4.9), (20000, 40.0, 4.0)])
def test_groups_accept_the_same_nodes(n, L, r_cut, theta, precision):
    """Few targets (one a warp) and all of them (groups): cutoff spheres that
    wrap around the box, opening angles below and above the cube diagonal."""
    x, y, z = points(n, L, 11)
    args = (r_cut / 4.5, r_cut, 0.05, theta, precision)
    every = np.arange(n, dtype=np.uint32)
    full = short_range_forces(L, x, y, z, 1.0, every, *args)
    few = np.arange(0, n, 16, dtype=np.uint32)
    one = short_range_forces(L, x, y, z, 1.0, few, *args)
    assert rel_rms([f[few] for f in full[:3]], one[:3]) <= SAME[precision]


@pytest.mark.parametrize("precision,ratio", [("fp64", 3.0), ("fp64", 4.5), ("fp64", 5.6), ("fp64", 7.0),
                                             ("fp32", 4.5), ("fp32", 6.0), ("fp32", 7.5), ("fp32", 10.5)])
def test_largest_group_on_a_handle_equals_single_targets(precision, ratio):
    """More than a million sources of a handle (groups of 16) against a sample
    walked one target a warp, at each polynomial degree and the closed form. The
    positions are multiples of 2^-32 L, which the precision form holds exactly."""
    n, L = 1000003, 128.0
    x, y, z = (np.floor(c / L * 2.0 ** 32) * (L / 2.0 ** 32) for c in points(n, L, 5))
    r_cut, eps = 5.5, 0.04
    r_s = r_cut / ratio
    few = np.arange(0, n, 1009, dtype=np.uint32)
    one = short_range_forces(L, x, y, z, 1.0, few, r_s, r_cut, eps, 0.5, precision)
    with hb.PMSolver(hb.MeshGeometry(L, 32), hb.PMForceMethod.treepm_long_range(r_s), precision) as s:
        s.upload(x, y, z, uniform_mass=1.0)
        full = s.treepm_short_forces(0.5, eps, r_cut)
    assert abs(full[3]["interactions_per_target"] - one[3]["interactions_per_target"]) \
        < 0.2 * one[3]["interactions_per_target"]
    assert rel_rms([f[few] for f in full[:3]], one[:3]) <= SAME[precision]


def tree_size(L, x, y, z):
    """(nodes, depth) from the definition: level by level, the runs of equal
    63-bit key prefixes whose parent run holds at least two sources."""
    def spread(v):
        v = v.astype(np.uint64)
        for s, k in ((32, 0x1f00000000ffff), (16, 0x1f0000ff0000ff), (8, 0x100f00f00f00f00f),
                     (4, 0x10c30c30c30c30c3), (2, 0x1249249249249249)):
            v = (v | (v << np.uint64(s))) & np.uint64(k)
        return v

    q = [np.minimum(np.floor(c / L * 2097152.0), 2097151).astype(np.uint64) for c in (x, y, z)]
    key = np.sort((spread(q[0]) << np.uint64(2)) | (spread(q[1]) << np.uint64(1)) | spread(q[2]))
    nodes, depth, parent_ok = 0, 0, np.ones(key.size, bool)
    for level in range(22):
        prefix = key >> np.uint64(3 * (21 - level))
        _, first, count = np.unique(prefix, return_index=True, return_counts=True)
        here = int(np.count_nonzero(parent_ok[first]))
        if here == 0:
            break
        nodes, depth = nodes + here, level
        parent_ok = np.repeat(count, count) >= 2
    return nodes, depth


@pytest.mark.parametrize("n,copies", [(2, 0), (3, 1), (255, 0), (256, 3), (257, 9), (1025, 40),
                                      (5000, 700)])
def test_tree_of_tile_edges_and_coincident_sources(oracle, n, copies):
    """Tiles of the node sweep around 256 sources; `copies` sources repeat others
    to the last bit (leaves of several sources at the deepest level) or up to a
    cell of the deepest levels. Node count and depth from the definition, forces
    from direct summation."""
    L, r_cut, eps = 20.0, 6.0, 0.02
    x, y, z = points(n, L, 100 + n)
    rng = np.random.default_rng(n)
    src, dst = rng.integers(0, n, copies), rng.permutation(n)[:copies]
    x[dst], y[dst], z[dst] = x[src], y[src], z[src]
    near = dst[::2]
    x[near] = np.mod(x[near] + L * rng.uniform(-3e-6, 3e-6, near.size), L)
    every = np.arange(n, dtype=np.uint32)
    got = short_range_forces(L, x, y, z, 1.0, every, r_cut / 4.5, r_cut, eps, 1e-6)
    assert (int(got[3]["nodes"]), int(got[3]["depth"])) == tree_size(L, x, y, z)
    ref = oracle.short_range_direct(L, x, y, z, 1.0, every, r_cut / 4.5, r_cut, eps)
    scale = max(float(np.max(np.abs(r))) for r in ref)
    assert max(float(np.max(np.abs(g - r))) for g, r in zip(got[:3], ref)) <= 1e-12 * max(scale, 1e-300)


def test_tree_of_tight_pairs_alone(oracle):
    """1000 pairs 1e-6 L apart: each hangs on a chain of single-child nodes, nine nodes
    a source in all. Node count from the definition, forces from direct summation."""
    L, r_cut, eps, n = 20.0, 6.0, 0.02, 1000
    rng = np.random.default_rng(8)
    first = rng.uniform(0.01 * L, 0.99 * L, (3, n))
    way = rng.normal(size=(3, n))
    second = first + 1e-6 * L * way / np.linalg.norm(way, axis=0)
    x, y, z = (np.concatenate([a, b]) for a, b in zip(first, second))
    every = np.arange(2 * n, dtype=np.uint32)
    got = short_range_forces(L, x, y, z, 1.0, every, r_cut / 4.5, r_cut, eps, 1e-6)
    assert (int(got[3]["nodes"]), int(got[3]["depth"])) == tree_size(L, x, y, z)
    assert got[3]["nodes"] > 6 * 2 * n + 64
    ref = oracle.short_range_direct(L, x, y, z, 1.0, every, r_cut / 4.5, r_cut, eps)
    assert rel_rms(got[:3], ref) <= TOL["fp64"]


def test_growing_tree_allocates_once():
    """One handle whose tree grows from solve to solve, as in a clustering run: after two
    solves the work arrays hold it (up to two nodes a source; once more for a tree beyond
    that), and the forces are those of a fresh handle, bit for bit."""
    L, side, r_s = 20.0, 27, 0.25
    n = side ** 3
    rng = np.random.default_rng(12)
    grid = (np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij")).reshape(3, n) + 0.5) * L / side
    grid += rng.uniform(-0.2, 0.2, (3, n)) * L / side
    clump = rng.uniform(0, L, (3, 40))[:, rng.integers(0, 40, n)] + rng.normal(0, 0.15, (3, n))
    pair = rng.uniform(0, L, (3, n))
    pair[:, 1::2] = pair[:, :n - 1:2] + 3e-6 * L * rng.uniform(-1, 1, (3, n // 2))
    states = [np.where(np.arange(n) < f * n, clump, grid) for f in (0.0, 0.2, 0.4, 0.6, 0.9)]
    states += [pair, pair, grid, pair]
    geometry, method = hb.MeshGeometry(L, 32), hb.PMForceMethod.treepm_long_range(r_s)
    made, nodes = [], []
    count = ctypes.c_uint64()
    with hb.PMSolver(geometry, method) as s:
        for p in states:
            x, y, z = np.mod(p, L)
            s.upload(x, y, z, uniform_mass=1.0)
            got = s.treepm_short_forces(0.5, 0.03, 4.5 * r_s)
            assert nat.lib().hyowon_pm_debug_tree_allocations(s.handle, ctypes.byref(count)) == 0
            made.append(count.value)
            nodes.append(got[3]["nodes"])
            with hb.PMSolver(geometry, method) as fresh:
                fresh.upload(x, y, z, uniform_mass=1.0)
                want = fresh.treepm_short_forces(0.5, 0.03, 4.5 * r_s)
            assert all(np.array_equal(g, w) for g, w in zip(got[:3], want[:3]))
    assert all(a < b for a, b in zip(nodes[:5], nodes[1:5])) and nodes[4] < 2 * n < nodes[5]
    assert made[1] == made[4], made          # grown trees of up to 2 n nodes
    assert made[6] == made[8], made          # beyond: one call past the block, one regrow
