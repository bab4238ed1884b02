"""Memory that only makes a skeleton faster (pools of shared tables and strata) finds no room on
the device: the call goes on without it."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
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


@pytest.mark.parametrize("name", ["FPGM_SET_POOL", "FPGM_STRATA_POOL"])
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


_CAPPED = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import fastpgm_gb300 as F
from oracle import oracle as O
raw, _, _ = F.generate(n_nodes=12, n_samples=100000, seed=31, n_edges=24, max_indegree=5, card=(4, 7))
cols, card = O.relabel(raw)
ref = O.pc_skeleton(cols, card, threads=16)
small, _, _ = F.generate(n_nodes=12, n_samples=12000, seed=31, n_edges=24, max_indegree=5, card=(4, 7))
scols, scard = O.relabel(small)
sref = O.pc_skeleton(scols, scard, threads=16)
batch = np.array([[0, 1, 2, 3, 4, 5, 6]] * 4, dtype=np.int32)

def learn(e, data, want):
    e.upload(data)
    st = e.pc_skeleton().to_dict()
    res = e.result()
    assert np.array_equal(res["adj"], want["adj"]) and res["sepsets"] == want["sepsets"]
    assert st["tests"] == want["stats"]["tests"] and st["large_tests"] > 0
    return st

if sys.argv[2] == "sizes":  # device memory of the per-test kernels on these samples, and a small skeleton's launches
    import torch
    with F.Engine(0) as e:  # loads the kernels
        e.upload(small)
        e.ci_test_batch(batch, 5)
    before = torch.cuda.mem_get_info()[0]
    with F.Engine(0) as e:
        e.upload(raw)
        e.ci_test_batch(batch, 5)
        print(before - torch.cuda.mem_get_info()[0])
    with F.Engine(0) as e:
        print(learn(e, small, sref)["kernel_launches"])
elif sys.argv[2] == "skeleton":
    with F.Engine(0) as e:
        for _ in range(2):
            learn(e, raw, ref)
        e.ci_test(0, 1, [2])  # a buffer of 128 MB more
else:
    with F.Engine(0) as e:
        e.upload(raw)
        e.ci_test_batch(batch, 5)  # the per-test kernels' memory
        learn(e, raw, ref)
        print(learn(e, small, sref)["kernel_launches"])
"""


def _run(what, cap=0, **more):
    env = dict(os.environ, FPGM_DEVICE_MEM_CAP=str(cap), **more)
    return subprocess.run([sys.executable, "-c", _CAPPED, ROOT, what], capture_output=True, text=True, env=env, timeout=600)


def _capped(what, cap=0, **more):
    out = _run(what, cap, **more)
    assert out.returncode == 0, (what, cap, out.stderr[-1500:])
    return [int(v) for v in out.stdout.split()]


@pytest.fixture(scope="module")
def sizes():
    held, launches = _capped("sizes")
    assert held > (1 << 30)
    return held, launches


@pytest.mark.parametrize("spare", [20, 60, 100, 160, 240, 500])
def test_pools_leave_room_for_what_a_skeleton_cannot_do_without(sizes, spare):
    """Device memory for the per-test kernels and some megabytes more, less than the strata's pool of
    8,192 sets asks for: a skeleton that succeeds without the pools succeeds with them, and so does a
    call after it that needs a buffer of its own."""
    cap = sizes[0] + (spare << 20)
    alone = _run("skeleton", cap, FPGM_SETS="0", FPGM_STRATA="0", FPGM_BOUND="0")
    if alone.returncode == 0:
        _capped("skeleton", cap)
    else:
        assert spare < 240 and "FPGM_DEVICE_MEM_CAP" in alone.stderr


def test_no_room_for_one_dataset_is_not_kept_for_the_next(sizes):
    """The strata's pool finds no room with the first dataset; a smaller one afterwards is counted as in
    an engine of its own."""
    assert _capped("later", sizes[0] + (500 << 20)) == [sizes[1]]
