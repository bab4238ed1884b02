"""P-values of the GPU's FP64 incomplete gamma (series and continued fraction) against the oracle's."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
import fastpgm_gb300 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("card,nz,scale", [(2, 0, 1), (3, 1, 1), (2, 5, 1), (7, 2, 1), (7, 2, 3), (5, 4, 1), (5, 4, 2)])
def test_device_p_value_matches_oracle(card, nz, scale):
    """df from 1 to ~10,000, G^2 on both sides of df (the function's two branches): every value
    is the FP64 one here.  Tolerance: exp(-x + a ln x - ln Gamma(a)) loses about a ln a ulps."""
    import torch
    rng = np.random.default_rng(17 * card + nz + scale)
    S, n = 40000, nz + 2
    cols = rng.integers(0, card, (n, S)).astype(np.uint8)
    if scale > 1:  # y copies x on part of the samples: G^2 well above df
        same = rng.random(S) < 0.02 * scale
        cols[nz + 1, same] = cols[nz, same]
    cols, cd = O.relabel(cols)
    pitch = (S + 15) // 16 * 16
    dev = torch.zeros((n, pitch), dtype=torch.uint8, device="cuda")
    dev[:, :S] = torch.from_numpy(cols).cuda()
    out = torch.zeros(ctypes.sizeof(F.CIResult), dtype=torch.uint8, device="cuda")
    z = np.arange(nz, dtype=np.int32)
    rc = F.load().fpgm_ci_test_noalloc(dev.data_ptr(), pitch, n, S, nz, nz + 1,
                                       z.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), nz, 0.05, 0, out.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream)
    assert rc == F.FPGM_OK
    r = F.CIResult.from_buffer_copy(out.cpu().numpy().tobytes())
    a = 0.5 * r.df
    tests = np.array([[nz, nz + 1, *z]], dtype=np.int32)
    exp = O.ci_tests(cols, cd, tests, nz, threads=1)[0].p_value
    assert r.rechecked == 1
    assert abs(r.p_value - exp) <= 4e-16 * (8 + a * max(1.0, np.log(a + 1)))


def test_single_test_leaves_the_process_sign_of_gamma_alone():
    """The host's part of a single test writes no state of the process (engines run on several
    threads): the C library's signgam keeps the value it had."""
    raw, _, _ = F.generate(n_nodes=6, n_samples=2000, seed=4, n_edges=8, max_indegree=3, card=(2, 4))
    signgam = ctypes.c_int.in_dll(ctypes.CDLL("libm.so.6"), "signgam")
    with F.Engine(0) as e:
        e.upload(raw)
        signgam.value = 77
        r = e.ci_test(0, 1, [2, 3])
        assert r.df > 0 and signgam.value == 77
