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


@pytest.mark.parametrize("scene,voxel", [
    ("plain_mc", 0.19),      # pencil beam, slots above 32 MB: copies of them
    ("ct", 0.21),            # rotating fan: groups of 2 slots of 25 MB
    ("ct", 0.18),            # 40 MB: four blocks per SM with one batch, one with many small ones
    ("phantom", 0.29),       # cone: groups of 3 slots of 21 MB
])
def test_totals_do_not_depend_on_the_slots_in_use(scene, voxel):
    from chatcarlo_b200 import phantoms as PH
    from chatcarlo_b200 import workloads as W
    from chatcarlo_b200.tally import VoxelGrid
    from chatcarlo_b200.transport import run_transport
    if scene == "phantom":
        raw, spec = PH.phantom(np.random.default_rng(1))
    else:
        raw, spec = {"ct": W.ct, "plain_mc": W.plain_mc}[scene](), {"ct": W.CT_GRID, "plain_mc": W.PLAIN_MC_GRID}[scene]
    shape = tuple(int(np.ceil(k * spec["voxel_cm"] / voxel)) for k in spec["shape"])
    res = []
    for b in (20_000, 2_900):
        g = VoxelGrid(origin_cm=np.asarray(spec["origin"], dtype=float), shape=shape, voxel_size_cm=voxel,
                      track_uncertainty=True)
        r = run_transport(raw, n_histories=20_000, seed=5, batch_size=b, dose_grid=True, grid_resolution_cm=voxel, grid=g)
        assert (g.n_batches, g.n_histories) == (-(-20_000 // b), 20_000)
        res.append((r, g))
    (r0, g0), (r1, g1) = res
    assert r0.fraction_absorbed == r1.fraction_absorbed and r0.n_voxel_visits == r1.n_voxel_visits
    for a, a0 in ((g1.kerma_keV, g0.kerma_keV), (g1.h10_track_pSv_cm3, g0.h10_track_pSv_cm3)):
        # additions of positive FP64 numbers, as above
        np.testing.assert_allclose(a, a0, rtol=2.0 ** -36, atol=0)
    np.testing.assert_allclose(g0.kerma_sum2, g0.kerma_keV ** 2 / 20_000, rtol=1e-14, atol=0)


def test_reset_clears_what_the_last_run_left():
    """Runs on one engine grid: batches folded away leave nothing to clear, a
    pending batch (photons scored without a fold) is cleared by the reset."""
    from chatcarlo_b200 import _native as N
    from chatcarlo_b200 import workloads as W
    from chatcarlo_b200.geometry import Geometry
    from chatcarlo_b200.transport import DeviceGrid, default_engine, run_transport
    eng = default_engine()
    raw, spec = W.plain_mc(), W.PLAIN_MC_GRID
    ref = run_transport(raw, n_histories=5_000, seed=3, dose_grid=True, grid=W.make_grid(spec)).grid
    host = W.make_grid(spec)
    geo = Geometry(raw["geometry"])
    ts, th = eng.tables(geo.materials(), need_muen=True)
    sh = eng.scene(geo, ts)
    dg = DeviceGrid(eng, host, stats=True)
    try:
        pos, d, e = W.pencil_beam_arrays(1_000, [0.0, 0.0, -20.0], [0.0, 0.0, 1.0], 60.0)
        edep = np.zeros(len(ts.names))
        N.check(eng.lib.cc_transport_photons(eng.ctx, sh, th, dg.handle, 1_000, N.dptr(pos), N.dptr(d), N.dptr(e), 1, 0,
                                             1, None, None, None, N.dptr(edep), None))
        dg.download(host)
        assert host.kerma_keV.sum() > 0                # pending
        dg.reset()
        dg.download(host)
        assert host.kerma_keV.max() == 0.0
    finally:
        dg.close()
        eng.lib.cc_scene_destroy(sh)
    again = run_transport(raw, n_histories=5_000, seed=3, dose_grid=True, grid=W.make_grid(spec)).grid
    np.testing.assert_allclose(again.kerma_keV, ref.kerma_keV, rtol=2.0 ** -36, atol=0)


@pytest.mark.parametrize("block", [32, 128, 160, 256])
def test_batch_groups_of_warps(block):
    """Blocks of one, four, five and eight warps, stepped in groups of four
    (enough histories per lane that they are): the same histories and scores."""
    from chatcarlo_b200 import phantoms as PH
    from chatcarlo_b200.batched import BatchedRun
    scenes, specs = PH.phantoms(3, 4, side=16, voxel_cm=2.0)
    got = []
    for shape in ({"block": 256, "blocks_per_sm": 3, "chunk": 256}, {"block": block, "blocks_per_sm": 1, "chunk": 64}):
        br = BatchedRun(scenes, specs, [70_000, 1, 120_001], shape=shape)
        counts, _ = br.run(seed=9)
        got.append((np.array(counts), [g.kerma_keV.copy() for g in br.download()]))
    assert np.array_equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1], got[1][1]):
        # additions of positive FP64 numbers, fewer than 2^20 per voxel
        np.testing.assert_allclose(b, a, rtol=2.0 ** -33, atol=0)


@pytest.mark.parametrize("dose_grid", [True, False])
def test_batch_size_above_the_histories_is_one_batch(dose_grid):
    """"Never split" values: one batch of all histories, whatever the size."""
    from chatcarlo_b200 import workloads as W
    from chatcarlo_b200.transport import run_transport
    n, res = 10_000, []
    for b in (10_000, 1_000_000, 10 ** 9):
        g = W.make_grid(W.ROOM_GRID) if dose_grid else None
        res.append((run_transport(W.room(), n_histories=n, seed=4, batch_size=b, dose_grid=dose_grid, grid=g), g))
    r0, g0 = res[0]
    for r, g in res:
        assert (r.n_batches, r.fraction_absorbed, r.n_voxel_visits) == (1, r0.fraction_absorbed, r0.n_voxel_visits)
        assert r.energy_deposited_MeV.keys() == r0.energy_deposited_MeV.keys()
        for k, v in r0.energy_deposited_MeV.items():
            # FP64 sums of at most 2^17 positive deposits each
            np.testing.assert_allclose(r.energy_deposited_MeV[k], v, rtol=2.0 ** -36, atol=0)
        if g is not None:
            assert (g.n_batches, g.n_histories) == (1, n) and np.array_equal(g.n_batches_hit, g0.n_batches_hit)
            for a, a0 in ((g.kerma_keV, g0.kerma_keV), (g.h10_track_pSv_cm3, g0.h10_track_pSv_cm3)):
                np.testing.assert_allclose(a, a0, rtol=2.0 ** -36, atol=0)
            np.testing.assert_allclose(g.kerma_sum2, g0.kerma_sum2, rtol=2.0 ** -34, atol=0)
