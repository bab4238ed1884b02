"""What a user of the engine has it do, as cases that can be timed and compared.

Sizes are those of the benchmark configurations (fastpgm_gb300/configs.py: c1 to c5), of the
tests, or generic ones between and beside them.  Samples are host arrays, as a user's program
has them after reading a file, except where the entry point takes device buffers.  Everything
is made from the seed: another seed is another random network and other samples of it.  A state keeps
the arrays that results are written to, as large as they can get; what a pass leaves of them
unwritten stays zero.
"""
import ctypes
import math

import numpy as np
import torch

import fastpgm_gb300 as F

ALPHA = 0.05


def listed():
    return [
        # one test asked interactively, or by a caller with a search of its own: the smallest call,
        # samples resident (37 variables, 5,000 samples: c1)
        dict(name="test_small", kind="test", nodes=37, samples=5000, indegree=1.25, indegree_max=4,
             card_lo=2, card_hi=4, dirichlet=1.0, tail=0, cond=2),
        # the same on a long dataset (c3's 500,000 samples)
        dict(name="test_long", kind="test", nodes=24, samples=500000, indegree=1.5, indegree_max=4,
             card_lo=3, card_hi=3, dirichlet=1.0, tail=0, cond=4),
        # one test on samples that another allocator holds on the device (50,000 samples: c2)
        dict(name="test_device", kind="device_test", nodes=100, samples=50000, indegree=2.0, indegree_max=5,
             card_lo=2, card_hi=5, dirichlet=0.5, tail=0, cond=3),
        # a batch of low-order tests, as a constraint-based search of the caller's own asks for
        dict(name="batch_low", kind="batch", nodes=100, samples=50000, indegree=2.0, indegree_max=5,
             card_lo=2, card_hi=5, dirichlet=0.5, tail=0, cond=1, tests=8192),
        # a batch of high-order tests on variables of many states: tables that are mostly empty
        dict(name="batch_high", kind="batch", nodes=150, samples=100000, indegree=1.3, indegree_max=3,
             card_lo=2, card_hi=8, dirichlet=0.3, tail=1, cond=5, tests=500),
        # whole structure learning (host samples in, skeleton and separating sets out), from the
        # smallest network in use to the largest: c1, an odd-sized one, c2, c3, c4
        dict(name="learn_c1", kind="learn", nodes=37, samples=5000, indegree=1.25, indegree_max=4, card_lo=2, card_hi=4,
             dirichlet=1.0, tail=0, depth=1000),
        dict(name="learn_odd", kind="learn", nodes=61, samples=20011, indegree=1.7, indegree_max=4,
             card_lo=2, card_hi=6, dirichlet=1.0, tail=0, depth=1000),
        dict(name="learn_c2", kind="learn", nodes=100, samples=50000, indegree=2.0, indegree_max=5,
             card_lo=2, card_hi=5, dirichlet=0.5, tail=0, depth=1000),
        dict(name="learn_c3", kind="learn", nodes=223, samples=500000, indegree=1.5, indegree_max=4,
             card_lo=3, card_hi=3, dirichlet=1.0, tail=0, depth=5),
        dict(name="learn_c4", kind="learn", nodes=1041, samples=100000, indegree=1.3, indegree_max=3,
             card_lo=2, card_hi=8, dirichlet=0.3, tail=1, depth=1000),
        # several independent datasets learnt together (c5's shape of job list, fewer and shorter jobs)
        dict(name="learn_jobs", kind="jobs", jobs=12, nodes_lo=20, nodes_hi=120, samples_lo=1000, samples_hi=40000,
             card_lo=2, card_hi=6, depth=1000),
        # parameters of a known network (job -j 1's second half) on c2's data
        dict(name="params_c2", kind="params", nodes=100, samples=50000, indegree=2.0, indegree_max=5,
             card_lo=2, card_hi=5, dirichlet=0.5, tail=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["test", "device_test", "batch", "learn", "learn", "learn", "jobs", "params"])
    lo = rng.choice([2, 2, 2, 3])
    c = dict(kind=kind, nodes=_log(rng, 20, 400), samples=_log(rng, 1000, 500000), indegree=rng.uniform(1.0, 2.0),
             indegree_max=rng.randint(3, 5), card_lo=lo, card_hi=lo + rng.randint(0, 4),
             dirichlet=rng.choice([0.3, 0.5, 1.0]), tail=0)
    if kind in ("test", "device_test"):
        c.update(nodes=_log(rng, 8, 100), cond=rng.randint(0, 4))
    elif kind == "batch":
        c.update(samples=_log(rng, 1000, 200000), cond=rng.randint(0, 6), tail=rng.choice([0, 0, 1]))
        # at most about a gigabyte of samples counted in one batch
        c["tests"] = max(16, min(_log(rng, 64, 16384), int(1.2e9 / c["samples"] / (1 + c["cond"]))))
    elif kind == "learn":
        # long datasets have few variables or a small depth, so that a pass stays below the largest listed one's
        c.update(samples=_log(rng, 1000, 250000), indegree=rng.uniform(1.0, 1.7), card_hi=lo + rng.randint(0, 3),
                 depth=rng.choice([3, 4, 5, 1000]))
        if c["samples"] > 30000:
            c["depth"] = min(c["depth"], 5)
            c["nodes"] = min(c["nodes"], 150)
    elif kind == "params":
        c["card_hi"] = min(c["card_hi"], 5)
    elif kind == "jobs":
        c = dict(kind="jobs", jobs=rng.randint(2, 12), nodes_lo=20, nodes_hi=rng.randint(30, 120), samples_lo=1000,
                 samples_hi=_log(rng, 2000, 40000), card_lo=2, card_hi=rng.randint(3, 6), depth=rng.choice([4, 1000]))
    return c


# ------------------------------------------------------------------ inputs
def _network(case, seed):
    """Host samples uint8 [variables, samples] of a random network, and its parents."""
    tail = (0.2, 9, 21) if case["tail"] else (0.0, 2, 2)
    cols, _, parents = F.generate(n_nodes=case["nodes"], n_samples=case["samples"], seed=1 + seed,
                                  avg_indegree=case["indegree"], max_indegree=case["indegree_max"], tail=tail,
                                  card=(case["card_lo"], case["card_hi"]), dirichlet=case["dirichlet"])
    return cols, parents


def _dense(cols):
    """The samples with each variable's ids in order of first appearance, and the state counts."""
    out, card = np.empty_like(cols), np.empty(len(cols), dtype=np.int64)
    for v, c in enumerate(cols):
        _, first, inv = np.unique(c, return_index=True, return_inverse=True)
        rank = np.empty(len(first), dtype=np.uint8)
        rank[np.argsort(first)] = np.arange(len(first), dtype=np.uint8)
        out[v], card[v] = rank[inv], len(first)
    return out, card


def _tests(case, seed, parents):
    """Rows x, y, z1..zd of distinct variables; every other pair is an arc of the network."""
    rng = np.random.default_rng(seed)
    n, m = case["nodes"], case.get("tests", 1)
    arcs = [(int(p), v) for v in range(n) for p in parents[v] if p >= 0]
    rows = np.empty((m, 2 + case["cond"]), dtype=np.int32)
    for t in range(m):
        x, y = arcs[rng.integers(len(arcs))] if arcs and t % 2 == 0 else rng.choice(n, 2, replace=False)
        z = [v for v in rng.permutation(n)[:2 + case["cond"]] if v != x and v != y][:case["cond"]]
        rows[t] = [x, y, *sorted(z)]
    return rows


def _job_specs(case, seed):
    rng = np.random.default_rng(case["jobs"])  # the sizes belong to the case, networks and samples to the seed
    specs = []
    for j in range(case["jobs"]):
        samples = math.exp(rng.uniform(math.log(case["samples_lo"]), math.log(case["samples_hi"])))
        specs.append(dict(n_nodes=int(rng.integers(case["nodes_lo"], case["nodes_hi"] + 1)), n_samples=int(samples),
                          avg_indegree=float(rng.uniform(1.5, 2.0)), max_indegree=5,
                          card=(case["card_lo"], case["card_hi"]), dirichlet=1.0, seed=1 + 1000 * seed + j))
    return specs


def _result(nodes):
    """Room for the skeleton of datasets of these many variables: adjacency, removed pairs, separating sets."""
    n, pairs = sum(nodes), sum(k * (k - 1) // 2 for k in nodes)
    return dict(adj=np.zeros((n, n), dtype=np.uint8), removed=np.zeros((pairs, 2), dtype=np.int32),
                sep_offsets=np.zeros(pairs + 1, dtype=np.int32), sep_vars=np.zeros(4 * pairs + 4096, dtype=np.int32))


def _parent_lists(parents):
    return [sorted(int(p) for p in row if p >= 0) for row in parents]


def _table_room(case):
    return case["nodes"] * case["card_hi"] ** (1 + case["indegree_max"])


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "jobs":
        s["data"] = [F.generate(**spec)[0] for spec in _job_specs(case, seed)]
        s.update(eng=F.Engine(0), lib=F.load(), **_result([len(c) for c in s["data"]]))
        return s
    cols, parents = _network(case, seed)
    if kind == "learn":
        s.update(eng=F.Engine(0), lib=F.load(), cols=cols, **_result([case["nodes"]]))
        return s
    if kind == "device_test":
        dense, _ = _dense(cols)
        pitch = (case["samples"] + 15) // 16 * 16
        dev = torch.zeros((case["nodes"], pitch), dtype=torch.uint8, device="cuda")
        dev[:, :case["samples"]] = torch.from_numpy(dense).cuda()
        row = _tests(case, seed, parents)[0]
        s.update(dev=dev, pitch=pitch, x=int(row[0]), y=int(row[1]), z=np.ascontiguousarray(row[2:]),
                 out=torch.zeros(ctypes.sizeof(F.CIResult) // 8, dtype=torch.float64, device="cuda"))
        s["lib"] = F.load()
        return s
    eng = F.Engine(0)
    eng.upload(cols)
    s["eng"] = eng
    if kind == "params":
        lists = _parent_lists(parents)
        s.update(lib=F.load(), offsets=np.cumsum([0] + [len(p) for p in lists]).astype(np.int32),
                 parents=np.array(sum(lists, []) + [0], dtype=np.int32),
                 tables=np.zeros(case["nodes"] + 1, dtype=np.int64), potentials=np.zeros(_table_room(case)))
    else:
        rows = _tests(case, seed, parents)
        s["tests"] = rows
        if kind == "test":
            s.update(x=int(rows[0, 0]), y=int(rows[0, 1]), z=[int(v) for v in rows[0, 2:]])
        else:
            s["lib"] = F.load()
    return s


# ------------------------------------------------------------------ passes
def run(s):
    return _RUN[s["case"]["kind"]](s)


def _check(lib, rc):
    if rc != F.FPGM_OK:
        raise F.FpgmError(rc, lib.fpgm_last_error().decode(errors="replace"))


def _run_test(s):
    r = s["eng"].ci_test(s["x"], s["y"], s["z"], alpha=ALPHA)
    return {"df": r.df, "independent": r.independent, "g2": np.float32(r.g2), "p": np.float32(r.p_value)}


_u8p, _i32p, _i64p, _f64p = (ctypes.POINTER(t) for t in (ctypes.c_uint8, ctypes.c_int32, ctypes.c_int64,
                                                         ctypes.c_double))
_CI = ctypes.sizeof(F.CIResult)
_FIELDS = np.dtype({"names": [f[0] for f in F.CIResult._fields_],
                    "formats": [np.dtype(f[1]) for f in F.CIResult._fields_],
                    "offsets": [getattr(F.CIResult, f[0]).offset for f in F.CIResult._fields_], "itemsize": _CI})


def _run_batch(s):
    # the C ABI's call: the records land in one array, with no Python object for each test
    rows = s["tests"]
    out = np.empty(len(rows), dtype=_FIELDS)
    lib = s["lib"]
    _check(lib, lib.fpgm_ci_test_batch(s["eng"]._h, rows.ctypes.data_as(_i32p), len(rows), rows.shape[1] - 2, ALPHA, 0,
                                       out.ctypes.data_as(ctypes.POINTER(F.CIResult))))
    # the statistic is a compensated FP32 sum, so it is given as what it is
    return {"df": out["df"], "independent": out["independent"], "g2": out["g2"].astype(np.float32),
            "p": out["p_value"].astype(np.float32)}


def _run_device_test(s):
    c, z, lib = s["case"], s["z"], s["lib"]
    _check(lib, lib.fpgm_ci_test_noalloc(s["dev"].data_ptr(), s["pitch"], c["nodes"], c["samples"], s["x"], s["y"],
                                         z.ctypes.data_as(_i32p), len(z), ALPHA, 0, s["out"].data_ptr(),
                                         torch.cuda.current_stream().cuda_stream))
    # this call's statistic and p-value are FP64; the whole numbers lie in the same record
    g2, df = F.CIResult.g2.offset // 8, F.CIResult.df.offset // 4
    return {"df_independent": s["out"].view(torch.int32)[df:df + 2], "g2_p": s["out"][g2:g2 + 2]}


def _skeleton(s, card):
    st = s["eng"].pc_skeleton(alpha=ALPHA, depth=s["case"]["depth"])
    # the C ABI's call, into arrays that the caller keeps
    h, lib, removed, variables = s["eng"]._h, s["lib"], ctypes.c_int32(), ctypes.c_int64()
    _check(lib, lib.fpgm_pc_result_sizes(h, None, ctypes.byref(removed), ctypes.byref(variables)))
    if variables.value > len(s["sep_vars"]):
        raise ValueError("%d separating variables: more than there is room for" % variables.value)
    _check(lib, lib.fpgm_pc_result_fetch(h, s["adj"].ctypes.data_as(_u8p), s["removed"].ctypes.data_as(_i32p),
                                         s["sep_offsets"].ctypes.data_as(_i32p), s["sep_vars"].ctypes.data_as(_i32p)))
    return {"adj": s["adj"], "removed": s["removed"], "sep_offsets": s["sep_offsets"], "sep_vars": s["sep_vars"],
            "card": card, "tests": np.array(st.tests, dtype=np.int64)}


def _run_learn(s):
    return _skeleton(s, s["eng"].upload(s["cols"]))


def _run_jobs(s):
    return _skeleton(s, np.concatenate(s["eng"].upload_jobs(s["data"])))


def _run_params(s):
    lib, pot = s["lib"], s["potentials"]
    _check(lib, lib.fpgm_mle_cpts(s["eng"]._h, s["offsets"].ctypes.data_as(_i32p), s["parents"].ctypes.data_as(_i32p),
                                  1, s["tables"].ctypes.data_as(_i64p), pot.ctypes.data_as(_f64p)))
    return {"potentials": pot, "tables": s["tables"]}


_RUN = {"test": _run_test, "batch": _run_batch, "device_test": _run_device_test, "learn": _run_learn,
        "jobs": _run_jobs, "params": _run_params}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: the samples a pass reads, once each, and its results.  Operations: one count per
    sample and test; structure learning tests every pair at least once, whatever the data."""
    kind = case["kind"]
    if kind == "jobs":
        specs = [(q["n_nodes"], q["n_samples"]) for q in _job_specs(case, 0)]
        return {"bytes": sum(n * S + n * n + 4.0 * n * (n - 1) for n, S in specs),
                "flops": sum(0.5 * n * (n - 1) * S for n, S in specs)}
    n, S = case["nodes"], case["samples"]
    if kind == "learn":
        return {"bytes": n * S + n * n + 8.0 * n * (n - 1) / 2, "flops": 0.5 * n * (n - 1) * S}
    if kind == "params":
        return {"bytes": n * S, "flops": float(n * S)}
    m = case.get("tests", 1)
    return {"bytes": min(n, m * (2 + case["cond"])) * S + m * _CI, "flops": float(m * S)}


# ------------------------------------------------------------------ 64-bit values
def _g2_of(cols, card, row):
    """df, G^2 and p of one test by the textbook formulas, in 64 bits; only observed strata."""
    x, y, z = int(row[0]), int(row[1]), [int(v) for v in row[2:]]
    code, size = np.zeros(cols.shape[1], dtype=np.int64), 1
    for v in z:
        code = code * int(card[v]) + cols[v]
        size *= int(card[v])
    if size > 1 << 18:
        _, code = np.unique(code, return_inverse=True)
        size = int(code.max()) + 1
    dx, dy = int(card[x]), int(card[y])
    t = np.bincount((code * dx + cols[x]) * dy + cols[y], minlength=size * dx * dy).reshape(size, dx, dy)
    nx, ny, nz = t.sum(2), t.sum(1), t.sum((1, 2))
    df = int(((np.maximum((nx > 0).sum(1), 1) - 1) * (np.maximum((ny > 0).sum(1), 1) - 1)).sum())
    k, i, j = np.nonzero(t)
    o = t[k, i, j].astype(np.float64)
    g2 = float(np.sum(2.0 * o * np.log(o * nz[k] / (nx[k, i].astype(np.float64) * ny[k, j]))))
    p = 1.0 if df == 0 else float(torch.special.gammaincc(torch.tensor(0.5 * df, dtype=torch.float64),
                                                         torch.tensor(0.5 * max(g2, 0.0), dtype=torch.float64)))
    return df, g2, p


def exact(case, seed):
    kind = case["kind"]
    if kind in ("learn", "jobs"):
        return None  # whole numbers only
    cols, parents = _network(case, seed)
    dense, card = _dense(cols)
    if kind == "params":
        out = []
        for v, lists in enumerate(_parent_lists(parents)):
            code, size = dense[v].astype(np.int64), 1
            for q in lists:
                code = code * int(card[q]) + dense[q]
                size *= int(card[q])
            n = np.bincount(code, minlength=int(card[v]) * size).reshape(int(card[v]), size).astype(np.float64)
            out.append(((n + 1.0) / (n.sum(0) + float(card[v]))).reshape(-1))
        pot = np.zeros(_table_room(case))
        pot[:sum(len(t) for t in out)] = np.concatenate(out)
        return {"potentials": pot, "tables": None}
    got = [_g2_of(dense, card, row) for row in _tests(case, seed, parents)]
    if kind == "device_test":
        return {"df_independent": None, "g2_p": np.array(got[0][1:])}
    g2, p = np.array([g[1] for g in got]), np.array([g[2] for g in got])
    if kind == "test":
        # p is 1 - CDF: below the CDF's own rounding it has no digits to compare
        return {"df": None, "independent": None, "g2": float(g2[0]), "p": float(p[0]) if p[0] > 1e-9 else None}
    return {"df": None, "independent": None, "g2": g2, "p": p}
