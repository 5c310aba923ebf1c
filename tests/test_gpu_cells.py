"""The near-field cell walk against an FP64 sum over every pair inside the cut.

Sizes and shapes where the batches of 32, the columns and the routing can go
wrong: a few particles, counts around a batch, boxes of three cuts, sparse
columns whose batches span the box, passes split among a block's warps and
whole ones, clumps that stay in the cell walk and clumps that go to the tree
walk, and several boxes (one without a cell grid) in one pass.
"""
import math
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "janus-sim_b200"))


def _erfc(x):
    return np.vectorize(math.erfc)(x)


def _short(pos, q, targets, L, r_s, rc, eps):
    """(force, sum of |pair force|, what pairs within 1e-5 of the cut carry, sum of
    |pair force| / r_p, pairs), per target."""
    out, mag, edge, grad, cnt = [], [], [], [], []
    for t in targets:
        d = pos - pos[t]
        d -= L * np.round(d / L)
        r2 = (d * d).sum(1)
        near = (r2 > 0) & (r2 < (rc * 1.00001) ** 2)
        d, r2, qj = d[near], r2[near], q[near]
        rp = np.sqrt(r2 + eps * eps)
        x = rp / (2 * r_s)
        f = np.sign(q[t]) * qj * (_erfc(x) + 2 / math.sqrt(math.pi) * x * np.exp(-x * x)) / rp ** 3 if len(x) else x
        r = np.sqrt(r2)
        at_cut = r > rc * 0.99999
        out.append((f[~at_cut, None] * d[~at_cut]).sum(0) if len(x) else np.zeros(3))
        mag.append((np.abs(f) * r).sum())
        edge.append((np.abs(f) * r)[at_cut].sum())
        grad.append(np.abs(f).sum())
        cnt.append(len(x))
    return np.array(out), np.array(mag), np.array(edge), np.array(grad), np.array(cnt)


def _bound(L, mag, edge, grad, cnt):
    """The table's entries are within 1.4e-5 of a pair's force; a sum of n terms
    rounds like 2^-24 sqrt(n) of their magnitudes (4 of these); scaled and shifted
    coordinates put 3 x 2^-24 L into each difference, and a pair's force F r / r_p^3
    moves by at most 3 F / r_p^3 per length."""
    eps = 2.0 ** -24
    return (1.4e-5 + 4 * eps * np.sqrt(cnt)) * mag + 9 * eps * L * grad + edge


def _points(kind, n, L, seed):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        x = (rng.random((n, 3)) - 0.5) * L
    elif kind == "line":       # one row of columns holds everything
        x = np.stack([(rng.random(n) - 0.5) * L, rng.normal(0.0, 0.01 * L, n), rng.normal(0.0, 0.01 * L, n)], 1)
    else:                      # a clump across the box's corner and a background
        c = rng.normal(0.0, 0.02 * L, (n - n // 4, 3)) + 0.5 * L
        x = np.concatenate([c, (rng.random((n // 4, 3)) - 0.5) * L])
    return (np.remainder(x + 0.5 * L, L) - 0.5 * L).clip(-0.49999 * L, 0.49999 * L).astype(np.float32)


# kind, n+, n-, L, PM grid, r_cut in units of r_s, theta
CASES = [
    ("uniform", 1, 0, 10.0, 16, 2.0, 0.5),
    ("uniform", 3, 2, 10.0, 16, 2.0, 0.5),
    ("uniform", 17, 15, 10.0, 16, 2.5, 0.5),
    ("uniform", 17, 16, 10.0, 16, 2.5, 0.5),
    ("uniform", 1500, 1301, 20.0, 16, 4.26, 0.5),       # just three cuts along the box
    ("uniform", 0, 5000, 50.0, 32, 4.5, 0.5),
    ("line", 700, 900, 40.0, 32, 4.5, 0.5),
    ("uniform", 150000, 160001, 80.0, 128, 4.5, 0.5),   # more batches than are split
    ("clump", 3000, 3000, 40.0, 64, 4.5, 0.5),          # stays in the cell walk
    ("clump", 90000, 90000, 40.0, 64, 4.5, 0.3),        # its dense blocks go to the tree walk
]


def _config(J, L, M, cut, theta, n):
    r_s = 1.25 * L / M
    return J.Config(box_L=L, pm_grid=M, theta=theta, softening=0.02 * L / max(n, 1) ** (1 / 3), r_s=r_s,
                    r_cut=cut * r_s, mu=3.0, G_mass_plus=1.0)


def _check(J, cfg, pp, pm, ap, am, multipoles, extra=None, seed=0):
    pos = np.concatenate([pp, pm]).astype(np.float64)
    mm = cfg.mu * len(pp) / len(pm) if len(pp) and len(pm) else cfg.mu
    q = np.concatenate([np.full(len(pp), 1.0), np.full(len(pm), -float(np.float32(mm)))])
    acc = np.concatenate([ap, am]).astype(np.float64)
    t = np.random.default_rng(seed).choice(len(pos), min(len(pos), 60), replace=False)
    f, mag, *rest = _short(pos, q, t, cfg.box_L, cfg.r_s, cfg.r_cut, cfg.softening)
    err = np.linalg.norm(acc[t] - f, axis=1)
    bound = _bound(cfg.box_L, mag, *rest) + (0.0 if extra is None else np.concatenate(extra)[t])
    if multipoles:   # nodes of the tree walk at this theta, against the force itself
        bound = bound + 5e-3 * np.linalg.norm(f, axis=1) + 1e-4 * np.median(mag)
    assert np.all(np.isfinite(acc)) and np.all(err <= bound + 1e-30), (err / np.maximum(bound, 1e-30)).max()


@pytest.mark.parametrize("kind,n_p,n_m,L,M,cut,theta", CASES)
def test_short_range_force(kind, n_p, n_m, L, M, cut, theta):
    import janus_treepm as J
    cfg = _config(J, L, M, cut, theta, n_p + n_m)
    pp, pm = _points(kind, n_p, L, 1), _points(kind, n_m, L, 2)
    s = J.Solver(cfg)
    s.set_state(pp, None, pm, None)
    ap, am = s.accel_part(J.JT_PART_SHORT)
    nodes = s.timings()["node_interactions"]
    s.close()
    assert (nodes > 0) == (kind == "clump" and n_p > 50000), nodes
    _check(J, cfg, pp, pm, ap, am, nodes > 0)


def test_boxes_of_every_route_in_one_pass():
    """Boxes without a cell grid (r_cut > L / 3), small and clustered ones share
    the pass's cell and batch tables.  The mesh part, taken out as a box alone
    computes it, leaves the pairs' force on every particle that is checked, inside
    the clumps and outside."""
    import janus_treepm as J
    rows = [CASES[4], ("uniform", 300, 200, 8.0, 16, 2.4, 0.0), CASES[9], CASES[1], CASES[8]]
    cfgs = [_config(J, L, M, cut, th, n_p + n_m) for _, n_p, n_m, L, M, cut, th in rows]
    cfgs[1].r_cut = 0.4 * cfgs[1].box_L
    B = J.Batch()
    pts = [(_points(k, n_p, L, 1), _points(k, n_m, L, 2)) for k, n_p, n_m, L, *_ in rows]
    ids = [B.add(c, pp, None, pm, None) for c, (pp, pm) in zip(cfgs, pts)]
    B.forces(ids, J.JT_PART_SHORT)
    B.forces(ids)                      # the second pass meets the first one's tables
    full = [B.accel(i) for i in ids]
    B.close()
    for row, c, (pp, pm), acc in zip(rows, cfgs, pts, full):
        s = J.Solver(c)
        s.set_state(pp, None, pm, None)
        mesh, alone = s.accel_part(J.JT_PART_PM), s.accel()
        s.close()
        tree = row is rows[2]
        short = [a.astype(np.float64) - m for a, m in zip(acc, mesh)]
        # the mesh force twice (32-bit FFTs): 1e-5 of its largest value in the box
        peak = max(float(np.abs(m).max()) for m in mesh if len(m))
        extra = [np.full(len(a), 1e-5 * peak) for a in acc]
        for seed in (0, 1):
            _check(J, c, pp, pm, *short, multipoles=tree or row is rows[1], extra=extra, seed=seed)
        for a, r in zip(acc, alone):
            if len(r):   # every particle, against its own force or the box's median
                size = np.linalg.norm(r.astype(np.float64), axis=1)
                diff = np.linalg.norm(a.astype(np.float64) - r, axis=1)
                assert np.all(diff <= 1e-4 * np.maximum(size, np.median(size))), (diff / np.maximum(size, np.median(size))).max()


def test_first_pass_of_a_large_clustered_box_counts_its_candidates():
    """The pass that times the column counts keeps its first run in a clustered
    box; that run's candidates are the pass's."""
    import janus_treepm as J
    n, L = 1 << 21, 100.0
    cfg = _config(J, L, 256, 4.5, 0.5, 2 * n)
    s = J.Solver(cfg)
    rng = np.random.default_rng(4)
    centres = (rng.random((512, 3)) - 0.5) * L   # not so dense that the tree walk takes them

    def points():
        x = centres[rng.integers(0, 512, n)] + rng.normal(0.0, 1.0, (n, 3))
        return (np.remainder(x + 0.5 * L, L) - 0.5 * L).clip(-0.49999 * L, 0.49999 * L).astype(np.float32)

    s.set_state(points(), None, points(), None)
    s.accel()
    first = s.timings()["candidates"]
    s.accel()
    again = s.timings()["candidates"]
    c = s.cells()
    s.close()
    assert c["reach"] > 2.0 * c["reach_uniform"] and c["to_tree"] == 0, c
    # the second pass's cells hold the same particles in another order
    assert again > 0 and abs(first - again) < 0.02 * again, (first, again)


@pytest.mark.parametrize("n,nb", [(20, 1), (300, 2), (1000, 3), (2500, 4), (4100, 5)])
def test_a_small_uniform_box_is_not_clustered(n, nb):
    """Every column of these boxes is in reach of every other, and counts once."""
    import janus_treepm as J
    cfg = _config(J, 20.0, 16, 4.1, 0.5, n)
    s = J.Solver(cfg)
    s.set_state(_points("uniform", n // 2, 20.0, 5), None, _points("uniform", n - n // 2, 20.0, 6), None)
    s.accel()
    c = s.cells()
    s.close()
    assert c["nb"] == nb and 2 * c["colm"] + 1 >= nb
    assert c["reach"] == c["reach_uniform"] == n and c["unscaled"] == 0 and c["to_tree"] == 0


def _box_with_clumps(n, L, clumps, per, seed):
    """n particles of one species, clumps x per / 2 of them in Gaussian clumps
    (0.3 wide, shared by the species), the rest uniform."""
    x = (np.random.default_rng(seed).random((n, 3)) - 0.5) * L
    c = (np.random.default_rng(99).random((clumps, 3)) - 0.5) * 0.9 * L
    m = clumps * per // 2
    x[:m] = c[np.arange(m) % clumps] + np.random.default_rng(seed + 1).normal(0.0, 0.3, (m, 3))
    return (np.remainder(x + 0.5 * L, L) - 0.5 * L).clip(-0.49999 * L, 0.49999 * L).astype(np.float32)


# particles per species, L, PM grid, clumps, particles in each, theta, tree walk
ROUTES = [
    (128 ** 3, 100.0, 256, 1, 200000, 0.5, True),     # 22 ms against 45 by the cell walk
    (128 ** 3, 100.0, 256, 1, 30000, 0.5, False),     # 4.3 ms against 6.6 by the tree walk
    (128 ** 3, 100.0, 256, 8, 50000, 0.5, True),
    (64 ** 3, 50.0, 128, 1, 200000, 0.0, False),      # no multipoles at theta 0
    (64 ** 3, 50.0, 128, 1, 200000, 0.8, True),
    (64 ** 3, 50.0, 128, 1, 1000, 0.8, False),
]


@pytest.mark.parametrize("n,L,M,clumps,per,theta,tree", ROUTES)
def test_route_of_clumps_in_a_uniform_box(n, L, M, clumps, per, theta, tree):
    """Massive clumps go to the tree walk and leave the rest of a uniform box to
    the cell walk; the forces of both are the pairs' (targets inside and outside)."""
    import janus_treepm as J
    r_s = 1.25 * L / M
    cfg = J.Config(box_L=L, pm_grid=M, theta=theta, softening=L / (2 * n) ** (1 / 3) / 30, r_s=r_s, r_cut=4.5 * r_s,
                   mu=19.0, G_mass_plus=1.0)
    pp, pm = _box_with_clumps(n, L, clumps, per, 1), _box_with_clumps(n, L, clumps, per, 5)
    s = J.Solver(cfg)
    s.set_state(pp, None, pm, None)
    ap, am = s.accel_part(J.JT_PART_SHORT)
    c = s.cells()
    s.close()
    assert (c["to_tree"] > 0) == tree and c["to_tree"] < 1.2 * clumps * per, c
    pos = np.concatenate([pp, pm]).astype(np.float64)
    q = np.concatenate([np.ones(n), np.full(n, -19.0)])
    acc = np.concatenate([ap, am]).astype(np.float64)
    rng = np.random.default_rng(0)
    inside = rng.integers(0, clumps * per // 2, 10)
    for t, multipoles in ((np.concatenate([inside, n + inside]), tree),
                          (rng.integers(n - n // 8, n, 10), False)):
        f, mag, *rest = _short(pos, q, t, L, r_s, cfg.r_cut, cfg.softening)
        err = np.linalg.norm(acc[t] - f, axis=1)
        # nodes at this theta: 5e-3 of the force, 1e-4 of what the clump's pairs add up to
        bound = _bound(L, mag, *rest) + (5e-3 * np.linalg.norm(f, axis=1) + 1e-4 * mag if multipoles else 0.0)
        assert np.all(err <= bound), (multipoles, (err / bound).max(), c)


def test_a_dense_clump_in_a_uniform_box_keeps_its_digits():
    """Targets inside a clump too small for the tree walk and for the box's mean to
    call it clustered: their differences are of unscaled positions and their sums
    run in chunks (scaled positions and running sums: 5e-5 of the force)."""
    import janus_treepm as J
    n, L, M, k = 64 ** 3, 50.0, 128, 12000
    r_s = 1.25 * L / M
    cfg = J.Config(box_L=L, pm_grid=M, softening=L / (2 * n) ** (1 / 3) / 30, r_s=r_s, r_cut=4.5 * r_s, mu=1.0,
                   G_mass_plus=1.0)
    pts = []
    for seed in (1, 2):
        x = (np.random.default_rng(seed).random((n, 3)) - 0.5) * L
        x[:k] = [20.3, -21.7, 19.1] + np.random.default_rng(seed + 10).normal(0.0, 0.1, (k, 3))
        pts.append(x.astype(np.float32))
    s = J.Solver(cfg)
    s.set_state(pts[0], None, pts[1], None)
    ap, _ = s.accel_part(J.JT_PART_SHORT)
    c = s.cells()
    s.close()
    assert c["to_tree"] == 0 and c["reach"] < 1.3 * c["reach_uniform"] and c["unscaled"] == 1, c
    pos = np.concatenate(pts).astype(np.float64)
    q = np.concatenate([np.ones(n), -np.ones(n)])
    t = np.arange(0, k, k // 60)
    f, mag, *_ = _short(pos, q, t, L, r_s, cfg.r_cut, cfg.softening)
    err = np.linalg.norm(ap[t] - f) / np.linalg.norm(f)
    # each pair rounded once or twice (2^-24), the table without bias; 1e-5 here
    assert err < 2.0 * 2.0 ** -24 * np.linalg.norm(mag) / np.linalg.norm(f), err


def test_opposite_species_at_one_point_in_a_clustered_box():
    """An m- particle on top of every m+ one takes exactly the opposite
    acceleration outside the crowded blocks, whichever batch either is in; inside,
    to the rounding of sums cut at different places."""
    import janus_treepm as J
    n, L, k = 60000, 40.0, 24000
    rng = np.random.default_rng(7)
    x = (rng.random((n, 3)) - 0.5) * L
    x[:k] = [12.0, 11.0, -13.0] + rng.normal(0.0, 0.8, (k, 3))
    x = x.astype(np.float32)
    s = J.Solver(J.Config(box_L=L, pm_grid=64, mu=3.0, softening=0.02))
    s.set_state(x, None, x.copy(), None)
    ap, am = s.accel_part(J.JT_PART_SHORT)
    c = s.cells()
    s.close()
    assert c["unscaled"] == 1 and c["to_tree"] == 0, c
    # blocks whose reach misses the clump (5 standard deviations and a block's side more)
    side = L / c["nb"]
    d = np.abs(x.astype(np.float64) - [12.0, 11.0, -13.0])
    far = (np.minimum(d, L - d) > (c["colm"] + 2) * side + 4.0).any(1)
    assert far.sum() > 10000
    assert np.array_equal(am[far], -ap[far]), (am[far] != -ap[far]).any(1).sum()
    assert np.abs(am + ap).max() <= 1e-5 * np.abs(ap).max()


def test_a_clustered_box_of_any_length_unit():
    """The same clustered box in units 2^57 times smaller (L = 5.8e18): the
    accelerations, scaled back, are the same up to the order of the sums."""
    import janus_treepm as J
    out = []
    for e in (0, 57):
        u = 2.0 ** e
        L = 40.0 * u
        x = [_points("clump", 4000, 40.0, seed) * np.float32(u) for seed in (1, 2)]
        cfg = J.Config(box_L=L, pm_grid=32, softening=0.02 * u, r_s=1.25 * L / 32, r_cut=4.5 * 1.25 * L / 32, mu=3.0,
                       G_mass_plus=2.0 ** (2 * e - 40 if e else 0))
        s = J.Solver(cfg)
        s.set_state(x[0], None, x[1], None)
        acc = np.concatenate(s.accel_part(J.JT_PART_SHORT)).astype(np.float64)
        assert s.cells()["unscaled"] == 1 and s.cells()["to_tree"] == 0
        s.close()
        out.append(acc * (2.0 ** 40 if e else 1.0))
    assert np.isfinite(out[1]).all()
    assert np.abs(out[1] - out[0]).max() <= 1e-5 * np.abs(out[0]).max()
