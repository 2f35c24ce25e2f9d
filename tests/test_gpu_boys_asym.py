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
