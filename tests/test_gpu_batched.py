"""Batched multi-scene runs: one launch over several scenes gives each scene
the same statistics as its own single-scene run, reproducibly."""
import numpy as np
import pytest

from chatcarlo_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from chatcarlo_b200.transport import default_engine
    return default_engine()


def _chi2(a, b, n_a, n_b, min_counts=50):
    """Per-voxel comparison of two kerma maps by their totals; the variance of
    each voxel's total is estimated from its batch statistics."""
    from chatcarlo_b200.tally import standard_error
    ma, mb = a.kerma_keV / n_a, b.kerma_keV / n_b
    sa = standard_error(a.kerma_keV, a.kerma_sum2, a.n_batches, a.n_histories)
    sb = standard_error(b.kerma_keV, b.kerma_sum2, b.n_batches, b.n_histories)
    with np.errstate(divide="ignore", invalid="ignore"):
        ok = (ma > 0) & (mb > 0) & (sa / ma < 0.2) & (sb / mb < 0.2)
    z = (ma[ok] - mb[ok]) / np.sqrt(sa[ok] ** 2 + sb[ok] ** 2)
    return float(np.mean(z ** 2)) if ok.any() else 0.0, int(ok.sum())


def test_batched_matches_single_scene_runs(engine):
    from chatcarlo_b200.batched import BatchedRun
    from chatcarlo_b200.transport import run_transport
    scenes, specs, _ = W.batched_scenes(n_scenes=5, seed=7)
    counts = [400_000] * 5
    br = BatchedRun(scenes, specs, counts, slots=20, engine=engine)
    try:
        sc, out = br.run(seed=11)
        grids = br.download()
        assert out.n_histories == sum(counts)
        for i, raw in enumerate(scenes):
            single = W.make_grid(specs[i])
            res = run_transport(raw, n_histories=counts[i], seed=50 + i, batch_size=counts[i] // 20,
                                dose_grid=True, grid=single, engine=engine)
            n = counts[i]
            for k, val in ((0, res.fraction_absorbed), (1, res.fraction_escaped)):
                p = sc[i, k] / n
                se = np.sqrt(max(p * (1 - p), 1e-12) / n + max(val * (1 - val), 1e-12) / n)
                assert abs(p - val) < 5 * se + 1e-9, (i, k, p, val)
            chi2, nv = _chi2(grids[i], single, n, n)
            if nv > 30:
                assert chi2 < 1.3, (i, chi2, nv)
    finally:
        br.close()


@pytest.mark.parametrize("fp32_cells,rtol", [(False, 1e-9), (True, 1e-4)])
def test_batched_replay_is_reproducible(engine, fp32_cells, rtol):
    """Same seed -> same counts; same kerma up to the order of the FP64
    additions with the default FP64 scratch cells, and of the FP32 ones with
    FP32 cells switched on."""
    from chatcarlo_b200.batched import BatchedRun
    scenes, specs, _ = W.batched_scenes(n_scenes=8, seed=3)
    counts = [int(x) for x in np.linspace(30_000, 300_000, 8)]
    engine.set_tally_fp32(fp32_cells)
    try:
        br = BatchedRun(scenes, specs, counts, slots=1, engine=engine)
    finally:
        engine.set_tally_fp32(False)
    try:
        a, _ = br.run(seed=5)
        ka = [g.kerma_keV.copy() for g in br.download()]
        br.reset()
        b, _ = br.run(seed=5)
        kb = [g.kerma_keV.copy() for g in br.download()]
        np.testing.assert_array_equal(a, b)
        for x, y in zip(ka, kb):
            np.testing.assert_allclose(x, y, rtol=rtol, atol=rtol * float(np.max(np.abs(y))))
        br.reset()
        c, _ = br.run(seed=6)
        assert not np.array_equal(a, c)
    finally:
        br.close()


def test_autotuner_picks_and_caches_a_shape(engine, tmp_path, monkeypatch):
    from chatcarlo_b200 import batched
    monkeypatch.setattr(batched, "CACHE_PATH", tmp_path / "autotune.json")
    scenes, specs, counts = W.batched_scenes(n_scenes=6, seed=9, hist_lo=2e4, hist_hi=1e5)
    cands = [{"block": 256, "blocks_per_sm": 2, "chunk": 128}, {"block": 256, "blocks_per_sm": 4, "chunk": 256}]
    shape = batched.autotune(scenes, specs, counts, engine=engine, scale=1.0, candidates=cands)
    assert shape in cands
    assert (tmp_path / "autotune.json").exists()
    assert batched.autotune(scenes, specs, counts, engine=engine, candidates=[]) == shape


HEEL_FIRST = """
import sys
import numpy as np
sys.path.insert(0, {root!r})
import chatcarlo_b200.source as S
from chatcarlo_b200 import phantoms as PH
from chatcarlo_b200.batched import BatchedRun
from chatcarlo_b200.transport import Engine
g = np.load({golden!r})
bins = (g["rect_centers"], tuple(zip(g["rect_spec_e"], g["rect_spec_w"])), g["rect_rel"], g["rect_rel"] * 1e6)
S.heel_spectra_for_source = lambda src, sid, span, n_bins=15: bins
scenes, specs = PH.phantoms(2, 4, side=32, voxel_cm=1.0)
heel = [dict(scenes[0], source={{"position": [0, -100, 0], "direction": [0, 1, 0], "heel_effect": True, "kvp": 80,
                                "field": {{"shape": "rect", "size_cm": [35, 43], "sid_cm": 100}},
                                "anode_direction": [1.0, 0.3, 0.0]}}), scenes[1]]
eng = Engine(0, precision="fp64")
ms, counts = [], []
for sc in (heel, scenes, heel):
    br = BatchedRun(sc, specs, [1_000_000] * 2, engine=eng)
    runs = [br.run(seed=1) for _ in range(24)]      # the first ones also bring the clocks up
    ms.append(min(o.elapsed_ms for _, o in runs[1:]))
    counts.append(runs[0][0])
    br.close()
assert np.array_equal(counts[0], counts[2]) and counts[0].sum() > 0
print(*ms)
"""


def test_a_heel_source_in_the_first_batch_of_a_process():
    """The FP64 engine's tallying batch asks for more than 48 KB of shared
    memory: the kernel with the heel effect gets the same launch (two blocks
    per SM, not one: 1.4 times the time) whether or not another batch ran before."""
    import subprocess
    import sys
    from conftest import GOLDEN, ROOT
    code = HEEL_FIRST.format(root=str(ROOT), golden=str(GOLDEN / "heel.npz"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    first, _, again = map(float, r.stdout.split())
    assert first < 1.1 * again, r.stdout


@pytest.mark.parametrize("scenes_n", [2, 9])
def test_scenes_that_share_a_grid_are_summed_once(engine, scenes_n):
    """One grid handle for several scenes holds the sum of their scores."""
    from chatcarlo_b200 import phantoms as PH
    from chatcarlo_b200.batched import BatchedRun
    scenes, specs = PH.phantoms(1, 4, side=48, voxel_cm=0.7)
    br = BatchedRun(scenes * scenes_n, specs * scenes_n, [30_000 + 1_000 * i for i in range(scenes_n)], engine=engine)
    try:
        br.run(seed=3)
        each = [(g.kerma_keV.copy(), g.h10_track_pSv_cm3.copy()) for g in br.download()]
        own = list(br.dgrids)
        br.dgrids = [own[0]] * scenes_n
        br._build()
        br.reset()
        for turns in (1, 2):
            br.run(seed=3)
            got = br.download()[0]
            for k, a in enumerate((got.kerma_keV, got.h10_track_pSv_cm3)):
                # FP64 additions of positive numbers, fewer than 2^17 per voxel
                np.testing.assert_allclose(a, turns * sum(e[k] for e in each), rtol=2.0 ** -36, atol=0)
        br.reset()
        assert br.download()[0].kerma_keV.max() == 0.0
        br.dgrids = own
    finally:
        br.close()


@pytest.mark.parametrize("batch_size", [5_000_000, 1_000])
def test_a_run_that_grows_a_grid_leaves_its_batch_usable(engine, batch_size):
    """A run on a batch's grid takes more scratch slots than the batch was
    captured with; both then add their scores to the grid."""
    from chatcarlo_b200 import _native as N
    from chatcarlo_b200 import phantoms as PH
    from chatcarlo_b200.batched import BatchedRun
    scenes, specs = PH.phantoms(2, 4, side=40, voxel_cm=0.8)
    scenes[0] = dict(scenes[0], source=dict(scenes[0]["source"], field={"shape": "parallel", "size_cm": [2.0, 2.0]}))
    br = BatchedRun(scenes, specs, [40_000, 50_000], engine=engine)
    out, edep = N.RunOut(), np.zeros(len(br.ts.names))

    def run_on_the_first_grid():
        N.check(engine.lib.cc_run(engine.ctx, br.scene_h[0], br.th, br.source_h[0], br.dgrids[0].handle, 20_000, batch_size,
                                  7, 0, 1, N.dptr(edep), None, out))

    def totals():
        return [g.kerma_keV.copy() for g in br.download()]

    try:
        br.run(seed=3)
        batch = totals()
        br.reset()
        run_on_the_first_grid()
        run = totals()
        assert run[0].sum() > 0 and run[1].max() == 0.0
        br.run(seed=3)
        for got, a, b in zip(totals(), run, batch):
            # FP64 additions of positive numbers, fewer than 2^17 per voxel
            np.testing.assert_allclose(got, a + b, rtol=2.0 ** -36, atol=0)
        br.reset()
        br.run(seed=3)
        for got, b in zip(totals(), batch):
            np.testing.assert_allclose(got, b, rtol=2.0 ** -36, atol=0)
    finally:
        br.close()
