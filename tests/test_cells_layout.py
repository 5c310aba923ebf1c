"""Host-side arithmetic of the near-field cell list, as the library computes it
(jt_cell_slot, jt_cell_layout): the slots that columns own for their batches of
32 never overlap and fit the table, and the columns a batch looks at cover the
cut on every side."""
import ctypes as C

import numpy as np
import pytest

import janus_treepm as J


def _slot(start, column, batch):
    out = C.c_int64()
    assert J.library().jt_cell_slot(int(start), int(column), int(batch), C.byref(out)) == J.JT_OK
    return out.value


@pytest.mark.parametrize("seed", range(6))
def test_batch_slots_are_disjoint_and_fit(seed):
    rng = np.random.default_rng(seed)
    counts = [rng.integers(0, 3, 400), rng.integers(0, 200, 300), np.full(50, 32), np.full(50, 33),
              np.where(rng.random(500) < 0.02, 5000, 0), np.array([1])][seed]
    start = np.concatenate([[0], np.cumsum(counts)])
    slots = []
    for c, n in enumerate(counts):
        slots += [_slot(start[c], c, k) for k in range((int(n) + 31) // 32)]
    assert len(slots) == len(set(slots))
    # the table ends where the column after the last would begin
    assert not slots or max(slots) < _slot(start[-1], len(counts), 0)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 65536, 600581, 22478848, 1 << 30])
@pytest.mark.parametrize("cuts", [2.9, 3.0003, 3.4, 4.9, 5.71, 11.4, 68.0, 400.0])
def test_columns_in_reach_cover_the_cut(n, cuts):
    L, rcut = 50.0, 50.0 / cuts
    cfg = J.Config(box_L=L, pm_grid=64, r_s=rcut / 4.5, r_cut=rcut, softening=0.01)
    o = J.cell_layout(cfg, n // 2, n - n // 2)
    nb, m = o["nb"], o["colm"]
    if cuts < 3.0:
        assert nb == 0                                 # the tree walk's box
        return
    side = L / nb
    assert 1 <= nb <= 256 and o["nbx"] == 8 * nb
    assert 1 <= m <= 2 and (2 * m + 1) ** 2 <= 32      # one lane per column
    assert m <= nb                                     # one wrap at most
    assert m * side >= rcut * 0.99999                  # column m + 1 lies beyond the cut
    assert nb == 1 or side ** 3 * n >= 31.99 * L ** 3  # a batch of 32 is no longer than its column is wide
    assert abs(o["reach_uniform"] - n * (min(2 * m + 1, nb) / nb) ** 3) <= 1e-6 * n


def test_bad_layouts_are_refused():
    o = J.jt_cell_info()
    bad = J.Config(box_L=50.0, pm_grid=33).to_c()
    assert J.library().jt_cell_layout(C.byref(bad), 10, 10, C.byref(o)) == J.JT_EINVAL
    assert J.library().jt_cell_slot(-1, 0, 0, C.byref(C.c_int64())) == J.JT_EINVAL
