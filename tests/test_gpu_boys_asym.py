"""The FP64 register evaluator of the Boys function (lgx_boys variant 1) beyond the
table's end, T > 50."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT_PI_2 = 0.88622692545275801365


@pytest.mark.parametrize("mmax", [0, 1, 2])
def test_f0_is_the_librarys_reciprocal_square_root(gpu_ctx, mmax):
    # sqrt(pi)/2 times CUDA's rsqrt (1 ulp over the whole range), rounded once: equal
    # to the last bit, up to the largest finite T (T to FP32 chooses the branch, so a
    # T within 2e-6 of 50 still takes the table)
    import torch
    rng = np.random.default_rng(8)
    T = np.concatenate([[50.001, 1e100, 1e300, np.finfo(float).max],
                        rng.uniform(50.001, 400.0, 20000), np.exp(rng.uniform(4.0, 700.0, 5000))])
    rs = torch.rsqrt(torch.from_numpy(T).cuda()).cpu().numpy()
    assert np.array_equal(gpu_ctx.boys(T, mmax, 1)[:, 0], ROOT_PI_2 * rs)


@pytest.mark.parametrize("mmax", [2, 3, 4, 5, 6])
def test_every_order_beyond_the_table(gpu_ctx, mmax):
    # F_0 carries rsqrt (2.2e-16 at most), the rounded constant and the product: 4.4e-16;
    # each step of the upward recursion the rounded square of rsqrt, the odd factor and
    # the product: 7.7e-16.  The dropped e^{-T} terms are below 2e-19 of F_6 from T = 60
    # on.  Up to T = 1e200, where F_0 is 1e-100 and the higher orders underflow.
    rng = np.random.default_rng(9)
    T = np.concatenate([rng.uniform(60.0, 300.0, 5000), 10.0 ** rng.uniform(2.0, 200.0, 5000)])
    F = gpu_ctx.boys(T, mmax, 1)
    L = np.longdouble
    want = np.sqrt(L(np.pi) / T.astype(L)) / 2
    want = want * np.sqrt(L("3.14159265358979323846264338327950288") / L(np.pi))
    for m in range(mmax + 1):
        err = np.abs(F[:, m].astype(L) - want)
        assert np.all(err <= L(4.4e-16 + 7.7e-16 * m + 1e-18) * want + L(5e-324) * (m + 1)), m
        want = want * (2 * m + 1) / (2 * T.astype(L))
