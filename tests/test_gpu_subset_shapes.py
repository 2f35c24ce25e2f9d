"""J/K passes over a pair subset: their launch shapes do not depend on the passes
that ran before on the same context (the shapes tuned for the full basis would
leave the subset's few quartets with serial chains), and neither do their results.

Bound: the same quartets in another order of the FP64 sums, 1e-12 of the largest
element."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_subset_pass_after_a_full_pass(lgx, mode):
    bs = lgx.BasisSet("cc-pVDZ", lgx.water_cluster(2, 2, 2))
    D = lgx.random_density(bs.nbf, 40, seed=5)
    pairs = [(i, j) for i in range(0, len(bs), 2) for j in range(0, i + 1, 2)]
    got = []
    for full_first in (True, False):
        ctx = lgx.Context(0)
        ctx.set_basis(bs)
        if full_first:
            ctx.jk(D, 1e-12, 0)
            ctx.jk(D, 1e-12, mode)
        ctx.set_pair_subset(pairs)
        J, K, _ = ctx.jk(D, 1e-12, mode)
        J, K, _ = ctx.jk(D, 1e-12, mode)  # the captured pass
        got.append((J, K, [(r["class"], r["fp32"], r["kernel"], r["shape"])
                           for r in ctx.last_pass_launches()]))
        ctx.close()
    (J, K, shapes), (J0, K0, shapes0) = got
    assert shapes == shapes0
    deep = [s for c, fp32, k, s in shapes if c == (0, 0, 0, 0) and not fp32]
    assert deep and deep[0] > 1
    assert np.max(np.abs(J - J0)) < 1e-12 * np.max(np.abs(J0))
    assert np.max(np.abs(K - K0)) < 1e-12 * np.max(np.abs(K0))
