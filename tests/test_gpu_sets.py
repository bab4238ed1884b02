"""Tests within shared memory scored from tables counted once per variable set (the default in
a skeleton) against the oracle and against tests that count their own (FPGM_SETS=0)."""
import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F

pytestmark = pytest.mark.gpu


def _skeleton(raw, depth=1000, alpha=0.05):
    with F.Engine(0) as e:
        e.upload(raw)
        st = e.pc_skeleton(alpha=alpha, depth=depth).to_dict()
        return st, e.result()


def _check(raw, depth=1000, alpha=0.05):
    cols, card = O.relabel(raw)
    ref = O.pc_skeleton(cols, card, alpha=alpha, depth=depth, threads=16)
    st, res = _skeleton(raw, depth, alpha)
    assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"]
    assert st["tests"] == ref["stats"]["tests"]
    return st


# samples: below one 16-sample vector, its edges, one warp's step and past it; cards: 32 copies
# of the smallest table down to one copy, then a CTA's tables (2,048 ints and more)
@pytest.mark.parametrize("n,S,card,edges", [(6, 9, (2, 2), 7), (8, 15, (2, 3), 10), (8, 16, (2, 3), 10),
                                            (10, 513, (2, 4), 14), (20, 1025, (2, 3), 30), (30, 4099, (2, 6), 45),
                                            (16, 30011, (2, 5), 30), (14, 20000, (7, 12), 16), (9, 50003, (15, 25), 9)])
def test_tables_per_set_match_oracle(n, S, card, edges):
    raw, _, _ = F.generate(n_nodes=n, n_samples=S, seed=S + n, n_edges=edges, max_indegree=4, card=card)
    _check(raw, depth=5)


@pytest.mark.parametrize("alpha", [0.0, 1e-5, 0.5, 1.0])
def test_tables_per_set_at_other_levels_of_significance(alpha):
    raw, _, _ = F.generate(n_nodes=14, n_samples=3000, seed=8, n_edges=20, max_indegree=4, card=(2, 4))
    _check(raw, depth=4, alpha=alpha)


@pytest.mark.parametrize("env", [{"FPGM_SETS": "0"}, {"FPGM_SET_POOL": "16"}, {"FPGM_SET_POOL": "20000"},
                                 {"FPGM_STRATA_POOL": "16"}, {"FPGM_STRATA_POOL": "900000"},
                                 {"FPGM_WARP_SLICE": "3072"}])
def test_out_of_room_counts_per_test(monkeypatch, env):
    """A pool of tables, or of stratum ids, that runs out: the tests left over count their own."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    raw, _, _ = F.generate(n_nodes=12, n_samples=12000, seed=31, n_edges=24, max_indegree=5, card=(4, 7))
    st = _check(raw)
    assert st["large_tests"] > 0


def test_constant_and_equal_columns():
    rng = np.random.default_rng(3)
    raw = rng.integers(0, 3, (9, 700)).astype(np.uint8)
    raw[2] = 0
    raw[5] = raw[4]
    raw[7] = (raw[1] + raw[6]) % 3
    _check(raw)


@pytest.mark.parametrize("bound", ["1", "0"])
@pytest.mark.parametrize("n,S,card,edges,alpha", [(40, 3000, (2, 3), 70, 0.05), (30, 20000, (2, 9), 45, 0.05),
                                                  (25, 4000, (2, 4), 60, 0.0), (25, 4000, (2, 4), 60, 0.9),
                                                  (20, 500, (2, 2), 40, 1e-4)])
def test_level_1_bounds_match_oracle(monkeypatch, bound, n, S, card, edges, alpha):
    """Level 1 decided from level 0's statistics where the chain rule allows (FPGM_BOUND=0: every
    test counted): near-copies of a variable put the bound close to the threshold."""
    monkeypatch.setenv("FPGM_BOUND", bound)
    raw, _, _ = F.generate(n_nodes=n, n_samples=S, seed=n + S, n_edges=edges, max_indegree=4, card=card)
    rng = np.random.default_rng(n)
    for v in range(0, n - 1, 5):  # noisy copies: strongly dependent pairs through a common neighbour
        keep = rng.random(S) < rng.uniform(0.05, 0.9)
        raw[v + 1, keep] = raw[v, keep]
    _check(raw, depth=4, alpha=alpha)


def test_level_1_bounds_across_datasets():
    data = [F.generate(n_nodes=n, n_samples=S, seed=S, n_edges=2 * n, max_indegree=4, card=(2, 5))[0]
            for n, S in ((12, 700), (30, 9000), (2, 40), (17, 2500))]
    with F.Engine(0) as e:
        e.upload_jobs(data)
        e.pc_skeleton()
        res = e.result()
        offsets = e.job_offsets
    for raw, (adj, seps) in zip(data, F.split_jobs(res, offsets)):
        cols, card = O.relabel(raw)
        ref = O.pc_skeleton(cols, card, threads=16)
        assert np.array_equal(adj, ref["adj"]) and seps == ref["sepsets"]


@pytest.mark.parametrize("pool", [None, "16", "20000"])
@pytest.mark.parametrize("n,S,card,edges,alpha", [(40, 3000, (2, 3), 70, 0.05), (30, 20000, (2, 9), 45, 0.05),
                                                  (25, 4000, (2, 4), 60, 0.0), (25, 4000, (2, 4), 60, 0.9),
                                                  (20, 15, (2, 3), 40, 0.3), (16, 9000, (11, 15), 20, 1e-4)])
def test_level_2_bounds_match_oracle(monkeypatch, pool, n, S, card, edges, alpha):
    """Level 2 decided from its sets of three variables at sizes below the rule's (FPGM_BOUND=2);
    sets whose tables found no room, or are past a warp's 2,048 cells, bound nothing."""
    monkeypatch.setenv("FPGM_BOUND", "2")
    if pool:
        monkeypatch.setenv("FPGM_SET_POOL", pool)
    raw, _, _ = F.generate(n_nodes=n, n_samples=S, seed=n + S, n_edges=edges, max_indegree=4, card=card)
    rng = np.random.default_rng(n)
    for v in range(0, n - 2, 4):  # noisy copies: dependence that one or two neighbours explain in part
        for k in (1, 2):
            keep = rng.random(S) < rng.uniform(0.05, 0.9)
            raw[v + k, keep] = raw[v, keep]
    _check(raw, depth=5, alpha=alpha)


def test_level_2_bounds_across_datasets(monkeypatch):
    monkeypatch.setenv("FPGM_BOUND", "2")
    data = [F.generate(n_nodes=n, n_samples=S, seed=S, n_edges=2 * n, max_indegree=4, card=(2, 5))[0]
            for n, S in ((12, 700), (30, 9000), (2, 40), (17, 2500))]
    with F.Engine(0) as e:
        for _ in range(2):  # the second pass finds the buffers of the first
            e.upload_jobs(data)
            e.pc_skeleton()
            res = e.result()
            for raw, (adj, seps) in zip(data, F.split_jobs(res, e.job_offsets)):
                cols, card = O.relabel(raw)
                ref = O.pc_skeleton(cols, card, threads=16)
                assert np.array_equal(adj, ref["adj"]) and seps == ref["sepsets"]
