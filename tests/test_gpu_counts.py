"""What a skeleton's counts read (fpgm_pc_stats count_bytes, large_bytes), by the way its tests are
counted, and with it which way that was: tables shared by variable set, shared strata, tests
decided by the bounds, and the per-test kernels that they all fall back to."""
import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F

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
