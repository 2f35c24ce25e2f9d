"""Mixed J/K passes with none, few, some and most of their quartets in FP32: the
launches of a pass with little FP32 work share all streams, the others split them
by precision.  Each threshold runs twice (launch by launch, then as the captured
graph) on one context against the FP64 pass.

Bound: an integral of an FP32 quartet is off by 1e-5 of its Schwarz bound at most
(test_gpu_configs.py), which lies below the threshold, times the density's elements;
the FP64 rest by the order of its sums, 1e-12 of the largest element."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis,waters", [("6-31G", (1, 1, 1)), ("cc-pVDZ", (2, 1, 1)),
                                          ("cc-pVTZ", (1, 1, 1))])
def test_mixed_passes_by_fp32_share(lgx, basis, waters):
    bs = lgx.BasisSet(basis, lgx.water_cluster(*waters))
    D = lgx.random_density(bs.nbf, 5 * waters[0], seed=3)
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    J, K, _ = ctx.jk(D, 1e-13, 0)
    shares = []
    for thr in (0.0, 1e-11, 1e-9, 1e-6, 1e-3, 1e-1):
        for _ in range(2):
            Jm, Km, st = ctx.jk(D, 1e-13, 1, thr)
            tol = 1e-5 * thr * np.abs(D).sum()
            assert np.max(np.abs(Jm - J)) <= tol + 1e-12 * np.max(np.abs(J))
            assert np.max(np.abs(Km - K)) <= tol + 1e-12 * np.max(np.abs(K))
        shares.append(st.quartets_fp32 / (st.quartets_fp32 + st.quartets_fp64))
    ctx.close()
    assert shares[0] == 0.0 and shares[-1] > 0.1 and shares == sorted(shares)
