"""The order in which a launch takes its histories, and the scratch copies of
a launch of few batches, change the order of FP64 additions only."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batches", [
    (1, (1, 200_000)),                      # one history: 31 lanes of its unit stay empty
    (33, (33, 7, 1)),                       # 1 batch in 16 copies; 5 batches in 2; 33 batches of one history
    (100_001, (200_000, 33_333, 7_001)),    # 1, 4 and 15 batches, the last one short
    (70_000, (1_000, 70_000)),              # 64 batches per launch, in groups of 16 and a short last launch
])
def test_totals_do_not_depend_on_the_batches(n, batches):
    from chatcarlo_b200 import workloads as W
    from chatcarlo_b200.transport import run_transport
    res = []
    for b in batches:
        g = W.make_grid(W.ROOM_GRID)
        r = run_transport(W.room(), n_histories=n, seed=11, batch_size=b, dose_grid=True, grid=g)
        res.append((b, r, g))
    _, r0, g0 = res[0]
    for b, r, g in res:
        nb = -(-n // b)
        assert (g.n_batches, g.n_histories) == (nb, n)
        assert r.fraction_absorbed == r0.fraction_absorbed and r.n_voxel_visits == r0.n_voxel_visits
        for a, a0 in ((g.kerma_keV, g0.kerma_keV), (g.h10_track_pSv_cm3, g0.h10_track_pSv_cm3)):
            # additions of positive FP64 numbers: at most 2^-53 of the sum each, fewer than 2^17 per voxel
            np.testing.assert_allclose(a, a0, rtol=2.0 ** -36, atol=0)
        assert np.array_equal(g.kerma_keV > 0, g0.kerma_keV > 0)
        assert g.n_batches_hit.max() <= nb and np.array_equal(g.n_batches_hit > 0, g.kerma_keV > 0)
        if nb == 1:
            np.testing.assert_allclose(g.kerma_sum2, g.kerma_keV ** 2 / n, rtol=1e-14, atol=0)
