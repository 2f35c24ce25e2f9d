"""The Boys evaluators of the mixed scheme's J/K kernels (lgx_boys variants 7
and 8: program and register kernels; 9: the register kernels' whole path from
primitive-pair data) against the oracle's F_m(T): T = 0, tiny, at and between
grid points, around the table's end at 50, and far beyond it.

Bound: one FP32 ulp, and the FP32 rounding of F_m itself for 99.5% of the values.
A value is one rounding of a leading FP32 part plus an FP32 correction below 2^-6
of it, whose own roundings move it by 2^-30 of F_m at most, 1/64 ulp; it rounds the
other way when it lies that close to a rounding boundary, which fewer than 1/64 of
the values do, and a quarter of that with the correction at its mean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TINY = np.finfo(np.float32).tiny


def _arguments():
    rng = np.random.default_rng(21)
    near = [np.nextafter(x, y) for x in (0.0, 25.0, 49.984375, 50.0, 50.015625) for y in (0, 99)]
    grid = np.arange(0, 50.02, 1.0 / 64)
    return np.concatenate([[0.0], near, np.exp(rng.uniform(np.log(1e-12), np.log(1.0), 300)), grid,
                           grid[:-1] + 1.0 / 128, rng.uniform(0, 50, 6000),
                           rng.uniform(49.9, 50.1, 500), rng.uniform(50, 120, 1500),
                           np.exp(rng.uniform(np.log(120), np.log(1e6), 500))])


def _check(F, ref):
    normal = np.abs(ref) >= TINY
    want, got = ref[normal].astype(np.float32), F[normal].astype(np.float32)
    ulps = np.abs(got.view(np.int32).astype(np.int64) - want.view(np.int32).astype(np.int64))
    assert ulps.max() <= 1 and np.mean(ulps == 0) > 0.995, (ulps.max(), np.mean(ulps == 0))
    assert np.all(F[~normal & (np.abs(ref) < 0.5 * TINY)] == 0.0)


@pytest.mark.parametrize("variant,mmax", [(7, 0), (7, 8), (7, 12), (8, 0), (8, 1), (8, 2), (8, 3),
                                          (8, 4), (8, 5), (8, 6)])
def test_jk_boys_is_rounded_to_fp32(gpu_ctx, oracle_mod, variant, mmax):
    T = _arguments()
    _check(gpu_ctx.boys(T, mmax, variant), np.array([oracle_mod.boys(float(t), mmax) for t in T]))


@pytest.mark.parametrize("mmax", [0, 1, 2, 4, 6])
def test_jk_register_path_from_pair_data(gpu_ctx, oracle_mod, mmax):
    rng = np.random.default_rng(31 + mmax)
    n = 6000
    zb, zk = np.exp(rng.uniform(np.log(0.05), np.log(3e4), (2, n)))
    Pb = rng.uniform(-30.0, 30.0, (n, 3))
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    d = np.exp(rng.uniform(np.log(1e-4), np.log(40.0), n))
    d[:50] = 0.0  # coincident centres: T = 0
    Pk = Pb + d[:, None] * u
    L = np.longdouble  # the argument from the same inputs in extended precision
    T = (zb.astype(L) * zk / (zb.astype(L) + zk) * ((Pb.astype(L) - Pk) ** 2).sum(1)).astype(float)
    assert (T > 50).sum() > 100 and (T < 1).sum() > 100
    _check(gpu_ctx.boys(np.column_stack([Pb, zb, Pk, zk]), mmax, 9),
           np.array([oracle_mod.boys(float(t), mmax) for t in T]))
