"""The FP64 core integrals of the attenuated operators as the register J/K kernels
form them (lgx_boys variant 10) against the same formulas in extended precision.

Bound: s = omega^2 / (omega^2 + rho) from a rounded sum and a rounded quotient and
its square root and powers, restated here step by step in FP64 with the Boys values
in extended precision, give the error that s brings; the evaluator (variant 1) adds
its own, which is measured on the same arguments, once for erf and twice for erfc.  The errors are independent
roundings, so their squares add; 10% over that sum covers the product and the
difference that neither holds.  Small T, where the powers of s are the whole of s's effect:
s taken from a reciprocal square root of omega^2 + rho has 1.4 to 1.8 times the
error there from m = 1 on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble


def _boys(T, mmax):
    """F_0..F_mmax in extended precision, 0 <= T <= 50: Maclaurin series of the
    top order, downward recursion."""
    T = T.astype(L)
    term = np.full_like(T, L(1) / (2 * mmax + 1))
    s = term.copy()
    for i in range(1, 400):
        term = term * (2 * T / (2 * mmax + 2 * i + 1))
        s = s + term
        if np.all(term < s * L(1e-21)):
            break
    e = np.exp(-T)
    F = [None] * (mmax + 1)
    F[mmax] = e * s
    for m in range(mmax - 1, -1, -1):
        F[m] = (2 * T * F[m + 1] + e) / (2 * m + 1)
    return np.array(F).T


def _core(op, s, root, G, F):
    """The formulas with the given s and sqrt(s), in the precision of s."""
    out, f = [], root
    for m in range(G.shape[1]):
        g = f * G[:, m].astype(s.dtype)
        out.append(g if op == "erf_coulomb" else F[:, m].astype(s.dtype) - g)
        f = f * s
    return np.array(out).T


@pytest.mark.parametrize("op", ["erf_coulomb", "erfc_coulomb"])
@pytest.mark.parametrize("mmax", [0, 2, 4, 6])
def test_attenuated_core_integrals(lgx, op, mmax):
    rng = np.random.default_rng(4)
    n, omega = 20000, 0.37
    rho = np.exp(rng.uniform(np.log(0.02), np.log(1e3), n))
    T = np.exp(rng.uniform(np.log(1e-4), np.log(2.0), n))
    ctx = lgx.Context(0)
    ctx.set_operator(lgx.Operator[op], omega)
    got = ctx.boys(np.column_stack([T, rho]), mmax, 10)
    own = ctx.boys(T, mmax, 1)
    ctx.close()
    w2 = omega * omega
    F = _boys(T, mmax)
    sl = L(w2) / (L(w2) + rho.astype(L))
    want = _core(op, sl, np.sqrt(sl), _boys(sl * T, mmax), F)
    s = w2 / (w2 + rho)
    emul = _core(op, s, np.sqrt(s), _boys(s * T, mmax), F)
    rms = lambda err, of: np.sqrt(np.mean((err / of).astype(float) ** 2, axis=0))
    e_own = rms(own - F, F) if op == "erf_coulomb" else np.sqrt(2) * rms(own - F, want)
    bound = 1.1 * np.sqrt(rms(emul - want, want) ** 2 + e_own ** 2)
    err = rms(got - want, want)
    assert np.all(err <= bound), (err / bound)


def test_attenuated_variant_needs_the_operator(gpu_ctx, lgx):
    with pytest.raises(lgx.LgxError):
        gpu_ctx.boys(np.array([[1.0, 1.0]]), 2, 10)
