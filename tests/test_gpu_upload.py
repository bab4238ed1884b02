"""Dataset upload, parameter tables and single tests at the edges of their kernels' splits: first-
appearance ids and cardinalities (one CTA or a cluster per column), parameter tables counted in
one or several slices, and single tests on one or several CTAs.  The expected values are NumPy's
and the oracle's; ids, counts and tables are compared exactly."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = F.Engine(0)
    yield e
    e.close()


def _columns(S, seed):
    """Columns of 1, 2, 31, 33 and 255 states (as far as S allows), a constant one, one whose only
    other value is the last sample, and one in descending order of first appearance."""
    rng = np.random.default_rng(seed)
    cols = [rng.integers(0, k, size=S) for k in (2, 31, 33, 255)]
    cols.append(np.full(S, 200))
    late = np.full(S, 7)
    late[-1] = 3
    cols.append(late)
    cols.append(np.maximum(0, 40 - np.arange(S)))
    return np.stack(cols).astype(np.uint8)


@pytest.mark.parametrize("S", [1, 15, 16, 17, 8191, 16383, 16384, 16385, 65536 + 5, 200003])
def test_relabel(eng, S):
    raw = _columns(S, S)
    want = np.empty_like(raw)
    states = []
    for v, c in enumerate(raw):
        _, first, inv = np.unique(c, return_index=True, return_inverse=True)
        rank = np.empty(len(first), dtype=np.uint8)
        rank[np.argsort(first)] = np.arange(len(first), dtype=np.uint8)
        want[v] = rank[inv]
        states.append(len(first))
    card = eng.upload(raw)
    assert np.array_equal(card, states)
    assert np.array_equal(eng.download(), want)
    # as given: the values stay and the cardinality is the largest + 1
    card = eng.upload(raw, relabel=False)
    assert np.array_equal(card, raw.max(axis=1).astype(int) + 1)
    assert np.array_equal(eng.download(), raw)


@pytest.mark.parametrize("S", [300, 40000])
def test_256_states_are_refused(eng, S):
    raw = np.zeros((3, S), dtype=np.uint8)
    raw[1] = np.arange(S) % 256
    with pytest.raises(F.FpgmError):
        eng.upload(raw)
    with pytest.raises(F.FpgmError):
        eng.upload(raw, relabel=False)


@pytest.mark.parametrize("S", [1, 15, 1025, 2048 * 16 + 3, 100007])
@pytest.mark.parametrize("card", [(2, 2), (3, 9)])
def test_parameter_tables(eng, S, card):
    """0 to 5 parents: one slice and several, byte and 16-bit codes, one and many replicas, tables
    of one entry per thread and of more configurations than threads."""
    raw, _, par = F.generate(n_nodes=12, n_samples=S, seed=5, n_edges=26, max_indegree=5, card=card)
    cols, states = O.relabel(raw)
    eng.upload(raw)
    parents = [par[v] for v in range(raw.shape[0])]
    got = eng.mle_cpts(parents, alpha=1)
    for v, (g, o) in enumerate(zip(got, O.mle_cpts(cols, states, parents, alpha=1))):
        assert g.shape == o.shape and np.array_equal(g, o), v


@pytest.mark.parametrize("S", [1, 15, 16, 4096, 8192, 40007])
def test_single_tests(eng, S):
    """fpgm_ci_test and its allocation-free form on one CTA and on several: counts, df and
    decisions equal to the oracle's, G^2 and p within the FP32 screen's bounds."""
    torch = pytest.importorskip("torch")
    lib = F.load()
    raw, _, _ = F.generate(n_nodes=10, n_samples=S, seed=17, n_edges=12, max_indegree=3, card=(2, 6))
    card = eng.upload(raw)
    cols = eng.download()
    pitch = (S + 63) // 64 * 64
    dev = torch.zeros((cols.shape[0], pitch), dtype=torch.uint8, device="cuda:0")
    dev[:, :S] = torch.from_numpy(cols)
    res = torch.zeros(ctypes.sizeof(F.CIResult), dtype=torch.uint8, device="cuda:0")
    rng = np.random.default_rng(S)
    for d in (0, 1, 2, 4):
        t = [int(v) for v in rng.choice(cols.shape[0], size=2 + d, replace=False)]
        want = O.ci_tests(cols, np.asarray(card, dtype=np.uint8), np.array([t], dtype=np.int32), d, threads=1)[0]
        z = np.array(t[2:] or [0], dtype=np.int32)
        rc = lib.fpgm_ci_test_noalloc(dev.data_ptr(), pitch, cols.shape[0], S, t[0], t[1],
                                      z.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), d, 0.05, 1, res.data_ptr(),
                                      None)
        assert rc == 0, lib.fpgm_last_error()
        torch.cuda.synchronize()
        for got in (F.CIResult.from_buffer_copy(res.cpu().numpy().tobytes()),
                    eng.ci_test(t[0], t[1], t[2:], want_hash=True)):
            assert got.table_hash == want.table_hash and got.cell_hash == want.cell_hash, t
            assert got.df == want.df and got.independent == want.independent, t
            assert abs(got.g2 - want.g2) <= max(2e-3, 2e-5 * abs(want.g2)), t
            assert abs(got.p_value - want.p_value) <= (1e-10 if got.rechecked else 1e-3), t
