"""Tests beyond shared memory counted through the variable sets they share (the default in a
skeleton) against the oracle and against the per-test kernels (FPGM_STRATA=0)."""
import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F

pytestmark = pytest.mark.gpu


def _skeleton(raw, depth=1000):
    with F.Engine(0) as e:
        e.upload(raw)
        st = e.pc_skeleton(depth=depth).to_dict()
        return st, e.result()


# samples: a multiple of 16 and the remainders beside it, below and past 2^16 (16-bit counters)
# and 2^17; cards: few strata (copies of the counters), many (rows taken in turns), past a
# mask word's 32 values (the per-test kernels); skew: one stratum with most of the samples
@pytest.mark.parametrize("S,card,edges,skew", [(5000, (6, 10), 24, 0.0), (20001, (5, 8), 30, 0.0),
                                               (20015, (3, 4), 34, 0.0), (70000, (6, 10), 30, 0.0),
                                               (66000, (12, 18), 30, 0.97), (140001, (6, 9), 20, 0.0),
                                               (9000, (28, 40), 12, 0.0)])
def test_shared_strata_match_oracle(monkeypatch, S, card, edges, skew):
    raw, _, _ = F.generate(n_nodes=12, n_samples=S, seed=S + card[1], n_edges=edges, max_indegree=5, card=card)
    if skew:  # most samples agree on every variable
        rng = np.random.default_rng(S)
        raw[:, rng.random(S) < skew] = 0
    cols, cd = O.relabel(raw)
    depth = 5 if card[0] > 20 else 1000
    ref = O.pc_skeleton(cols, cd, depth=depth, threads=16)
    st, res = _skeleton(raw, depth)
    assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"]
    assert st["tests"] == ref["stats"]["tests"]
    monkeypatch.setenv("FPGM_STRATA", "0")
    st0, res0 = _skeleton(raw, depth)
    assert st["large_tests"] == st0["large_tests"] > 0
    assert st["tests_executed"] == st0["tests_executed"]


def test_shared_strata_across_datasets():
    """Several datasets in one engine: their sets share the trie, their samples differ."""
    data = [F.generate(n_nodes=n, n_samples=S, seed=S, n_edges=2 * n, max_indegree=5, card=(4, 8))[0]
            for n, S in ((10, 3000), (14, 20011), (9, 66001))]
    with F.Engine(0) as e:
        e.upload_jobs(data)
        st = e.pc_skeleton().to_dict()
        res = e.result()
        offsets = e.job_offsets
    assert st["large_tests"] > 0
    for raw, (adj, seps) in zip(data, F.split_jobs(res, offsets)):
        cols, card = O.relabel(raw)
        ref = O.pc_skeleton(cols, card, threads=16)
        assert np.array_equal(adj, ref["adj"]) and seps == ref["sepsets"]


@pytest.mark.parametrize("alpha", [0.0, 1e-4, 0.3, 0.99, 1.0])
def test_shared_strata_at_other_levels_of_significance(alpha):
    raw, _, _ = F.generate(n_nodes=10, n_samples=12000, seed=5, n_edges=20, max_indegree=5, card=(5, 8))
    cols, card = O.relabel(raw)
    ref = O.pc_skeleton(cols, card, alpha=alpha, depth=5, threads=16)
    with F.Engine(0) as e:
        e.upload(raw)
        st = e.pc_skeleton(alpha=alpha, depth=5).to_dict()
        res = e.result()
    assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"]
    assert st["tests"] == ref["stats"]["tests"]
