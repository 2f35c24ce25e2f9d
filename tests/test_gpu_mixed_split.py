"""The mixed scheme's J/K kernels with the split-table Boys function: every
class from (ss|ss) to (ff|ff) in FP32 against the same pass in FP64, at
distances that put the Boys argument at zero, between grid points, around the
table's end (T = 50) and far beyond it.

Bound: an FP32 value passes through at most ~100 roundings of 2^-24 (prefactor,
recurrences up to L = 12, transform, digestion), 6e-6 of the largest terms; the
terms of one element of J or K are bounded by the largest element within a
factor of a few for the positive density used: 3e-5 of max |J|, |K|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax", [1, 3])
@pytest.mark.parametrize("dist", [0.0, 0.11, 6.9, 7.1, 40.0])
def test_mixed_split_boys_vs_fp64(lgx, lmax, dist):
    # exponents 2 on both centres: rho = 2 for the one-centre pairs, T = 2 R^2:
    # 95.2 and 100.8 at 6.9 / 7.1, and T = 50 lies between the mixed-pair
    # arguments (rho 1.1 and 0.4) there
    shells = []
    for c in (0.0, dist):
        for l in range(lmax + 1):
            shells.append(lgx.Shell(l, [(2.0, 0.7), (0.4, 0.5)], [c, 0.3 * c, 0.0], pure=l > 1))
    bs = lgx.BasisSet(shells)
    n = bs.nbf
    rng = np.random.default_rng(3)
    A = rng.uniform(0.0, 1.0, (n, n))
    D = np.eye(n) + 0.5 / n * (A + A.T)
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    J, K, _ = ctx.jk(D, 1e-14, 0)
    Jm, Km, st = ctx.jk(D, 1e-14, 1, 1e30)
    assert st.quartets_fp32 > 0 and st.quartets_fp64 == 0
    assert np.max(np.abs(Jm - J)) < 3e-5 * np.max(np.abs(J))
    assert np.max(np.abs(Km - K)) < 3e-5 * np.max(np.abs(K))
    ctx.close()
