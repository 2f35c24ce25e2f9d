"""Single shell sets of the register classes (one quartet over several blocks)
against the same quartet through the program kernel: primitive counts around a
warp, a block and the largest grid, every side that a pair or the bra and ket can
be swapped to, first derivatives, and a quartet whose primitives are all dropped.

Bound: the same FP64 terms of up to 65536 primitive quartets, summed in another
order: 65536 roundings of 1.1e-16 at worst, 1e-11 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shells(lgx, ls, ns, far=0.0):
    rng = np.random.default_rng(sum(ns) + 7 * sum(ls))
    out = []
    for k, (l, n) in enumerate(zip(ls, ns)):
        ex = np.exp(rng.uniform(np.log(0.3), np.log(9.0), n))
        out.append(lgx.Shell(l, list(zip(ex, rng.uniform(0.2, 1.0, n))),
                             rng.uniform(-1.2, 1.2, 3) + far * k, pure=l > 1))
    return out


def _both(lgx, monkeypatch, shells, deriv):
    res = []
    for off in ("0", "1"):
        monkeypatch.setenv("LGX_DISABLE_RK", off)
        ctx = lgx.Context(0)
        e = lgx.Engine(lgx.Operator.coulomb, 16, 3, deriv, context=ctx)
        r = e.compute(*shells)
        again = e.compute(*shells)  # the ticket is back at zero
        assert (r is None) == (again is None)
        if r is not None:
            assert np.array_equal(np.stack(r), np.stack(again))
            r = np.stack(r)
        res.append(r)
        ctx.close()
    return res


@pytest.mark.parametrize("ns", [(1, 1, 2, 1), (2, 4, 4, 1), (3, 11, 1, 1), (2, 8, 8, 1),
                                (10, 13, 1, 1), (4, 8, 8, 8), (16, 16, 16, 16)])
@pytest.mark.parametrize("ls,deriv", [((0, 0, 0, 0), 0), ((1, 1, 1, 1), 0), ((0, 2, 1, 0), 0),
                                      ((3, 0, 0, 1), 0), ((0, 1, 1, 0), 1), ((1, 0, 1, 1), 1)])
def test_one_quartet_vs_program_kernel(lgx, monkeypatch, ls, deriv, ns):
    a, b = _both(lgx, monkeypatch, _shells(lgx, ls, ns), deriv)
    assert np.max(np.abs(a - b)) < 1e-11 * np.max(np.abs(b))


@pytest.mark.parametrize("deriv", [0, 1])
def test_one_quartet_screened_out(lgx, monkeypatch, deriv):
    a, b = _both(lgx, monkeypatch, _shells(lgx, (1, 0, 1, 0), (3, 5, 2, 7), far=40.0), deriv)
    assert a is None and b is None
