"""Memory that only makes a skeleton faster (pools of shared tables and strata) finds no room on
the device: the call goes on without it."""
import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F

pytestmark = pytest.mark.gpu

MORE_THAN_ANY_GPU = str(1 << 50)


def _check(eng, raw, ref):
    eng.upload(raw)
    st = eng.pc_skeleton().to_dict()
    res = eng.result()
    assert np.array_equal(res["adj"], ref["adj"]) and res["sepsets"] == ref["sepsets"]
    assert st["tests"] == ref["stats"]["tests"]
    return st


@pytest.mark.parametrize("name", ["FPGM_SET_POOL"])
def test_pool_that_cudaMalloc_refuses(monkeypatch, name):
    """cudaMalloc's own refusal (not the engine's cap, which never reaches it) is no error of the
    call: the tests count their own tables."""
    monkeypatch.setenv(name, MORE_THAN_ANY_GPU)
    raw, _, _ = F.generate(n_nodes=12, n_samples=12000, seed=31, n_edges=24, max_indegree=5, card=(4, 7))
    cols, card = O.relabel(raw)
    ref = O.pc_skeleton(cols, card, threads=16)
    with F.Engine(0) as e:
        for _ in range(2):
            assert _check(e, raw, ref)["large_tests"] > 0
