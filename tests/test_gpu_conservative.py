"""Conservative primitive screening of single shell sets: the register kernels
against the block kernel, at coarse precisions where the two estimates (|pfac|
alone, and with the non-spherical factors and the number of primitive quartets)
keep different primitive quartets.

Bound: both keep the same primitive quartets (one screen, the same FP64 values) and
sum the same terms in another order: up to 1296 roundings of 1.1e-16, 1e-12 of the
largest value.  A primitive quartet that only one of them kept would count for the
precision's order, 1e-9 and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shells(lgx, ls, n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for l in ls:
        ex = np.exp(rng.uniform(np.log(0.08), np.log(40.0), n))
        out.append(lgx.Shell(l, list(zip(ex, rng.uniform(0.1, 1.0, n))),
                             rng.uniform(-2.0, 2.0, 3), pure=l > 1))
    return out


def _compute(lgx, monkeypatch, off, shells, deriv, precision, method):
    monkeypatch.setenv("LGX_DISABLE_RK", off)
    ctx = lgx.Context(0)
    e = lgx.Engine(lgx.Operator.coulomb, 16, 3, deriv, precision=precision, screening=method,
                   context=ctx)
    r = e.compute(*shells)
    ctx.close()
    return None if r is None else np.stack(r)


@pytest.mark.parametrize("n", [1, 2, 6])
@pytest.mark.parametrize("precision", [1e-4, 1e-6])
@pytest.mark.parametrize("ls,deriv", [((1, 1, 1, 1), 0), ((2, 1, 0, 0), 0), ((0, 2, 1, 0), 0),
                                      ((2, 0, 2, 0), 0), ((3, 0, 1, 0), 0), ((1, 0, 1, 1), 1)])
def test_conservative_register_vs_block_kernel(lgx, monkeypatch, ls, deriv, precision, n):
    differ = 0
    for seed in range(6):
        sh = _shells(lgx, ls, n, seed)
        a = _compute(lgx, monkeypatch, "0", sh, deriv, precision, lgx.ScreeningMethod.Conservative)
        b = _compute(lgx, monkeypatch, "1", sh, deriv, precision, lgx.ScreeningMethod.Conservative)
        o = _compute(lgx, monkeypatch, "1", sh, deriv, precision, lgx.ScreeningMethod.Original)
        assert (a is None) == (b is None)
        if b is None:
            continue
        assert np.max(np.abs(a - b)) < 1e-12 * np.max(np.abs(b))
        differ += o is None or not np.array_equal(o, b)
    assert n < 6 or differ  # the inputs do tell the two methods apart
