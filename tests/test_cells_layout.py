"""Host-side arithmetic of the near-field cell list, restated: the slots that
columns own for their batches of 32 never overlap and fit the table, and the
columns a batch looks at cover the cut on every side (jt_walk.cu
k_cell_scatter / k_walk_cell, jt_batch.cu cell_columns / box_cells)."""
import numpy as np
import pytest


@pytest.mark.parametrize("seed", range(6))
def test_batch_slots_are_disjoint_and_fit(seed):
    rng = np.random.default_rng(seed)
    counts = [rng.integers(0, 3, 400), rng.integers(0, 200, 300), np.full(50, 32), np.full(50, 33),
              np.where(rng.random(500) < 0.02, 5000, 0), np.array([1])][seed]
    start = np.concatenate([[0], np.cumsum(counts)])
    slots = []
    for c, n in enumerate(counts):
        slots += [(int(start[c]) >> 5) + c + k for k in range((int(n) + 31) // 32)]
    assert len(slots) == len(set(slots))
    assert not slots or max(slots) < int(start[-1]) // 32 + len(counts)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 65536, 600581, 22478848, 1 << 30])
@pytest.mark.parametrize("cuts", [3.0003, 3.4, 4.9, 5.71, 11.4, 68.0, 400.0])
def test_columns_in_reach_cover_the_cut(n, cuts):
    L, rcut = 1.0, 1.0 / cuts
    nb = int(max(1.0, min(256.0, L / np.cbrt(32.0 / n), 1.9 * L / rcut)))
    m = int(rcut * 1.0001 * nb / L + 1.0e-4) + 1
    side = L / nb
    assert 1 <= m <= 2 and (2 * m + 1) ** 2 <= 32      # one lane per column
    assert m <= nb                                     # one wrap at most
    assert m * side >= rcut * 0.99999                  # column m + 1 lies beyond the cut
