"""The tiled deposit and interpolation against the FP64 mesh of the same scheme
(oracle/acc_pm.c): tiles of 8^3 and 16^3 cells and passes that mix edges,
crowded tiles (a warp per particle) beside sparse ones, every assignment order
with and without interlacing, empty species; and a screened box's two sources
against an unscreened one in the limit of a long screening length."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path[:0] = [os.path.join(ROOT, "janus-sim_b200"), os.path.join(ROOT, "oracle")]

# PM grid, n+, n-, share of the particles in a clump across a tile corner, order, interlace
CASES = [
    (8, 40, 30, 0.0, 4, 1),        # one tile
    (16, 300, 0, 0.0, 3, 1),
    (32, 700, 900, 0.0, 4, 1),     # 8 tiles of 16^3: taken as 64 of 8^3
    (32, 3000, 2500, 0.95, 4, 1),  # crowded tiles among them
    (32, 3000, 2500, 0.95, 2, 2),
    (32, 3000, 2500, 0.95, 3, 1),
    (64, 4000, 4100, 0.9, 4, 2),   # tiles of 16^3
    (64, 0, 2049, 1.0, 4, 1),      # around the bound of a crowded tile
    (64, 2048, 0, 1.0, 4, 1),
]


def _points(n, share, L, M, seed):
    rng = np.random.default_rng(seed)
    k = int(share * n)
    # about one cell wide, a quarter cell off the corner of 8 tiles (of either edge)
    clump = rng.normal(0.0, 0.7 * L / M, (k, 3)) + 0.25 * L / M
    x = np.concatenate([clump, (rng.random((n - k, 3)) - 0.5) * L])
    return (np.remainder(x + 0.5 * L, L) - 0.5 * L).clip(-0.49999 * L, 0.49999 * L).astype(np.float32)


def _config(J, M, order, interlace):
    L = 2.0 * M
    return J.Config(box_L=L, pm_grid=M, softening=0.05, r_s=1.25 * L / M, r_cut=2.5 * 1.25 * L / M, mu=3.0,
                    G_mass_plus=1.0, pm_order=order, pm_interlace=interlace)


def _exact(O, cfg, pp, pm):
    pos = np.concatenate([pp, pm]).astype(np.float64)
    mm = cfg.mu * len(pp) / len(pm) if len(pp) and len(pm) else cfg.mu
    mass = np.concatenate([np.full(len(pp), 1.0), np.full(len(pm), mm)])
    sg = np.concatenate([np.ones(len(pp), np.int8), -np.ones(len(pm), np.int8)])
    return O.acc_pm_forces(pos, mass, sg, cfg.pm_grid, cfg.box_L, cfg.r_s, order=cfg.pm_order,
                           interlace=cfg.pm_interlace == 1)


def _close(got, ref):
    # single-precision FFTs and sums of up to 64 x 2 terms: 1e-5 of the largest force
    assert np.all(np.isfinite(got))
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max(), np.abs(got - ref).max() / np.abs(ref).max()


@pytest.mark.parametrize("M,n_p,n_m,share,order,interlace", CASES)
def test_mesh_force(M, n_p, n_m, share, order, interlace):
    import janus_treepm as J
    import oracle as O
    cfg = _config(J, M, order, interlace)
    pp, pm = _points(n_p, share, cfg.box_L, M, 1), _points(n_m, share, cfg.box_L, M, 2)
    s = J.Solver(cfg)
    s.set_state(pp, None, pm, None)
    got = np.concatenate(s.accel_part(J.JT_PART_PM)).astype(np.float64)
    s.close()
    _close(got, _exact(O, cfg, pp, pm))


def test_mixed_tile_edges_in_one_pass():
    import janus_treepm as J
    import oracle as O
    B, want, ids = J.Batch(), [], []
    for M, n_p, n_m, share, *_ in (CASES[0], CASES[3], CASES[6], (128, 500, 400, 0.0, 4, 1)):
        cfg = _config(J, M, 4, 1)
        pp, pm = _points(n_p, share, cfg.box_L, M, 1), _points(n_m, share, cfg.box_L, M, 2)
        ids.append(B.add(cfg, pp, None, pm, None))
        want.append((cfg, pp, pm))
    for _ in range(2):             # the second time from the sorted state
        B.forces(ids)
        full = [np.concatenate(B.accel(i)).astype(np.float64) for i in ids]
    B.close()
    for (cfg, pp, pm), got in zip(want, full):
        s = J.Solver(cfg)
        s.set_state(pp, None, pm, None)
        short = np.concatenate(s.accel_part(J.JT_PART_SHORT)).astype(np.float64)
        s.close()
        ref = _exact(O, cfg, pp, pm)
        assert np.abs(got - short - ref).max() <= 1e-5 * (np.abs(ref).max() + np.abs(short).max())


@pytest.mark.parametrize("M", [32, 64, 256])
def test_screened_sources_in_the_long_limit(M):
    """kappa -> 0: the two sources' forces add up to the unscreened one's."""
    import janus_treepm as J
    cfg = _config(J, M, 4, 1)
    pp, pm = _points(3000, 0.8, cfg.box_L, M, 1), _points(2500, 0.8, cfg.box_L, M, 2)
    out = []
    for lam in (0.0, 1.0e7):
        s = J.Solver(cfg)
        s.set_state(pp, None, pm, None)
        if lam:
            s.set_screening(lam)
        out.append(np.concatenate(s.accel()).astype(np.float64))
        s.close()
    _close(out[1], out[0])
