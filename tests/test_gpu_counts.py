"""What a skeleton's counts read (fpgm_pc_stats count_bytes, large_bytes), by the way its tests are
counted, and with it which way that was: tables shared by variable set, shared strata, tests
decided by the bounds, and the per-test kernels that they all fall back to."""
import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F
from fastpgm_gb300 import configs as C
from test_gpu_fullsize import check_job, fixture

pytestmark = pytest.mark.gpu


def _skeleton(monkeypatch, raw, ref=None, depth=1000, passes=1, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with F.Engine(0) as e:
        for _ in range(passes):
            e.upload(raw)
            st = e.pc_skeleton(depth=depth).to_dict()
            if ref is not None:
                res = e.result()
                assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"]
                assert st["tests"] == ref["stats"]["tests"]
    for k in env:
        monkeypatch.delenv(k)
    return st


@pytest.fixture(scope="module")
def mixed():
    """Tables on both sides of shared memory's size."""
    raw, _, _ = F.generate(n_nodes=12, n_samples=12000, seed=31, n_edges=24, max_indegree=5, card=(4, 7))
    cols, card = O.relabel(raw)
    return raw, O.pc_skeleton(cols, card, threads=16)


def test_shared_tables_count_their_columns_once(monkeypatch, mixed):
    raw, ref = mixed
    alone = _skeleton(monkeypatch, raw, ref, FPGM_SETS="0")["count_bytes"]
    assert _skeleton(monkeypatch, raw, ref, FPGM_SET_POOL="16")["count_bytes"] == alone
    assert 0 < _skeleton(monkeypatch, raw, ref)["count_bytes"] < alone


def test_shared_strata_count_their_sweeps(monkeypatch, mixed):
    raw, ref = mixed
    alone = _skeleton(monkeypatch, raw, ref, FPGM_STRATA="0")
    assert _skeleton(monkeypatch, raw, ref, FPGM_STRATA_POOL="16")["large_bytes"] == alone["large_bytes"]
    shared = _skeleton(monkeypatch, raw, ref)
    assert 0 < shared["large_bytes"] != alone["large_bytes"] and shared["large_tests"] == alone["large_tests"]


def _copies(n, S, card, edges, seed, step=5, reach=1):
    """Noisy copies of a variable: dependence that a neighbour or two explain in part."""
    raw, _, _ = F.generate(n_nodes=n, n_samples=S, seed=seed, n_edges=edges, max_indegree=4, card=card)
    rng = np.random.default_rng(n)
    for v in range(0, n - reach, step):
        for k in range(1, reach + 1):
            keep = rng.random(S) < rng.uniform(0.05, 0.9)
            raw[v + k, keep] = raw[v, keep]
    return raw


def test_level_1_bounds_leave_tests_uncounted(monkeypatch):
    """Without shared tables every counted test reads its own columns: fewer bytes are fewer counts."""
    raw = _copies(40, 3000, (2, 3), 70, 3040)
    cols, card = O.relabel(raw)
    ref = O.pc_skeleton(cols, card, depth=2, threads=16)
    got = {b: _skeleton(monkeypatch, raw, ref, depth=2, FPGM_SETS="0", FPGM_BOUND=b) for b in ("1", "0")}
    assert got["1"]["tests_executed"] == got["0"]["tests_executed"]
    assert 0 < got["1"]["count_bytes"] < got["0"]["count_bytes"]


def test_level_1_bounds_leave_tests_uncounted_across_datasets(monkeypatch):
    data = [_copies(n, S, (2, 4), 2 * n, S + n) for n, S in ((30, 3000), (20, 2500))]
    got = {}
    for bound in ("1", "0"):
        monkeypatch.setenv("FPGM_BOUND", bound)
        with F.Engine(0) as e:
            e.upload_jobs(data)
            st = e.pc_skeleton(depth=2).to_dict()
            got[bound] = st["count_bytes"], st["tests_executed"]
    assert got["1"][1] == got["0"][1] and 0 < got["1"][0] < got["0"][0]


@pytest.mark.parametrize("pool", [None, "16"])
def test_level_2_bounds_leave_tests_uncounted(monkeypatch, pool):
    """FPGM_BOUND=2 bounds level 2 at this size too, 1 does not; with no room for level 1's tables
    there is nothing to bound it by."""
    raw = _copies(40, 3000, (2, 3), 70, 3040, step=4, reach=2)
    cols, card = O.relabel(raw)
    ref = O.pc_skeleton(cols, card, depth=3, threads=16)
    env = {"FPGM_SET_POOL": pool} if pool else {}
    got = {b: _skeleton(monkeypatch, raw, ref, depth=3, FPGM_BOUND=b, **env)["count_bytes"] for b in ("2", "1")}
    assert got["2"] == got["1"] if pool else 0 < got["2"] < got["1"]


# ------------------------------------------------------------------ the per-test kernels of large tables
@pytest.fixture(scope="module")
def large():
    """Levels 6 to 9 partition half of their tests or more, the last three after a level of the same."""
    raw, _, _ = F.generate(n_nodes=24, n_samples=50000, seed=72, n_edges=70, max_indegree=6, card=(4, 7))
    cols, card = O.relabel(raw)
    return raw, O.pc_skeleton(cols, card, threads=16)


# from level 2 on, whatever the measured fraction (the fraction is measured on tests that a CTA keeps)
_BITMAPS = {"FPGM_LIVE_FRAC": "1.01", "FPGM_LIVE_MIN_LEVEL": "2", "FPGM_WIDE": "0"}


@pytest.mark.parametrize("env", [{}, {"FPGM_OVF_SKIP": "0"}, {"FPGM_STAGE_REC": "64"}, {"FPGM_STAGE_REC": "1024"},
                                 {"FPGM_LIVE": "0"}, _BITMAPS, {**_BITMAPS, "FPGM_STAGE_REC": "512"},
                                 {**_BITMAPS, "FPGM_GRAPH": "0"}])
def test_large_tables_test_by_test(monkeypatch, capfd, large, env):
    """A skeleton without shared strata (FPGM_STRATA=0): hashed, staged and partitioned strata and the
    contributing-sample bitmaps, three skeletons on one engine.  Every test reads its own columns.  The wave
    log, which takes the same path, shows partitioned tests and the levels that wrote bitmaps."""
    raw, ref = large
    st = _skeleton(monkeypatch, raw, ref, passes=3, FPGM_STRATA="0", **env)
    assert st["large_tests"] > 0 and st["large_bytes"] % raw.shape[1] == 0
    capfd.readouterr()
    log = _skeleton(monkeypatch, raw, ref, passes=1, FPGM_WAVE_LOG="1", **env)
    lines = capfd.readouterr().err.splitlines()
    assert log["large_bytes"] == st["large_bytes"]
    assert sum(int(w.split("(partitioned=")[1].split()[0]) > 0 for w in lines if "(partitioned=" in w) >= 4
    wrote = [int(w.split("level=")[1].split()[0]) for w in lines if w.startswith("live ") and " wrote=1 " in w]
    assert wrote == ([6, 7, 8, 9] if "FPGM_LIVE_FRAC" in env else [])


def test_bitmaps_of_a_larger_dataset_test_by_test(monkeypatch, capfd, large):
    """Bitmap pools of 30,000 samples remade for 50,000 in one engine."""
    small, _, _ = F.generate(n_nodes=24, n_samples=30000, seed=72, n_edges=70, max_indegree=6, card=(5, 9))
    cols, card = O.relabel(small)
    for k, v in {**_BITMAPS, "FPGM_WAVE_LOG": "1"}.items():
        monkeypatch.setenv(k, v)
    with F.Engine(0) as e:
        for raw, ref in ((small, O.pc_skeleton(cols, card, threads=16)), large):
            e.upload(raw)
            for _ in range(2):
                st = e.pc_skeleton().to_dict()
                res = e.result()
                assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"]
                assert st["tests"] == ref["stats"]["tests"]
            assert " wrote=1 " in capfd.readouterr().err


def test_full_size_skeleton_test_by_test(monkeypatch):
    """1,041 variables x 100,000 samples without shared strata: bitmaps by their default rule, tests scored
    by several CTAs."""
    fx = fixture("c4")
    raw, depth, _ = C.make_config("c4")
    monkeypatch.setenv("FPGM_STRATA", "0")
    with F.Engine(0) as e:
        e.upload(raw)
        st = e.pc_skeleton(depth=depth).to_dict()
        res = e.result()
    assert st["tests"] == fx["jobs"][0]["tests"] and st["large_bytes"] % raw.shape[1] == 0 and st["tune_timed"] > 0
    check_job(res["adj"], res["sepsets"], fx["jobs"][0])


# ------------------------------------------------------------------ edges of the rules
def test_strata_rows_of_wide_counters(monkeypatch):
    """A stratum of more than 65,535 samples beside more (stratum, value) cells than 32-bit counters
    fit shared memory at once: rows of wide counters taken in turns."""
    raw, _, _ = F.generate(n_nodes=8, n_samples=200000, seed=9, n_edges=14, max_indegree=4, card=(12, 18))
    rng = np.random.default_rng(9)
    raw[:, rng.random(raw.shape[1]) < 0.5] = 0
    cols, card = O.relabel(raw)
    ref = O.pc_skeleton(cols, card, depth=4, threads=16)
    shared = _skeleton(monkeypatch, raw, ref, depth=4)
    alone = _skeleton(monkeypatch, raw, ref, depth=4, FPGM_STRATA="0")
    assert shared["large_tests"] == alone["large_tests"] > 0 and shared["large_bytes"] != alone["large_bytes"]


@pytest.mark.parametrize("card", [(2, 4), (8, 12)])
def test_samples_at_the_fixed_point_limit(monkeypatch, card):
    """2^20 samples are the most that are decided in fixed point; one more takes the FP32 screen, level 0
    on the tensor cores included.  One engine, to and fro: its table of n ln n and the unit stay right."""
    raw, _, _ = F.generate(n_nodes=6, n_samples=(1 << 20) + 1, seed=20, n_edges=9, max_indegree=3, card=card)
    depth = 1000 if card[0] < 8 else 4
    bytes_read = {}
    for env in ({}, {"FPGM_SETS": "0", "FPGM_STRATA": "0", "FPGM_BOUND": "0"}):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        with F.Engine(0) as e:
            for S in (5000, 1 << 20, (1 << 20) + 1, 1 << 20):
                part = np.ascontiguousarray(raw[:, :S])
                cols, cd = O.relabel(part)
                ref = O.pc_skeleton(cols, cd, depth=depth, threads=16)
                e.upload(part)
                st = e.pc_skeleton(depth=depth).to_dict()
                res = e.result()
                assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"], S
                assert st["tests"] == ref["stats"]["tests"], S
                bytes_read[bool(env), S] = st["count_bytes"] + st["large_bytes"]
    assert bytes_read[False, (1 << 20) + 1] == bytes_read[True, (1 << 20) + 1]
    assert bytes_read[False, 1 << 20] != bytes_read[True, 1 << 20]


def test_datasets_past_the_fixed_point_limit():
    """Several datasets, one of them longer than the limit: level 0 on the counting kernels in FP32."""
    data = [F.generate(n_nodes=n, n_samples=S, seed=S, n_edges=n + 3, max_indegree=3, card=(2, 4))[0]
            for n, S in ((6, (1 << 20) + 17), (9, 3000))]
    with F.Engine(0) as e:
        e.upload_jobs(data)
        e.pc_skeleton()
        for raw, (adj, seps) in zip(data, F.split_jobs(e.result(), e.job_offsets)):
            cols, card = O.relabel(raw)
            ref = O.pc_skeleton(cols, card, threads=16)
            assert np.array_equal(adj, ref["adj"]) and seps == ref["sepsets"]
