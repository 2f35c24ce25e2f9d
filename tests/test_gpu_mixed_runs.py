"""FP32 quartets of deep contractions in a mixed J/K pass, one lane to a quartet:
(ab|00) of s shells with eight primitives each, 4096 primitive quartets, against
FP64.

Bound: the sum is taken in runs of 128 and over the 32 runs, 160 additions of a sum
that grows evenly: each rounds by 2^-24/sqrt(3) of the running sum at most (root
mean square), together sqrt(160/3) times that, 2.5e-7; the FP32 transform, density
and digestion add less than 1e-7: 3.5e-7 root mean square over the integrals.  One
run of 4096 gives 1.4e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2])
def test_deep_fp32_sums(lgx, monkeypatch, mode):
    monkeypatch.setenv("LGX_TUNE", "0")  # the default shape: one lane where quartets fill the GPU
    rng = np.random.default_rng(0)
    shells = [lgx.Shell(0, list(zip(np.exp(rng.uniform(np.log(0.3), np.log(9.0), 8)),
                                    rng.uniform(0.2, 1.0, 8))), rng.uniform(-0.02, 0.02, 3),
                        pure=False)
              for _ in range(26)]
    bs = lgx.BasisSet(shells)
    D = np.zeros((26, 26))
    D[0, 0] = 1.0
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    J, _, _ = ctx.jk(D, 0.0, 0)
    Jm, _, _ = ctx.jk(D, 0.0, mode, 1e30)
    assert [r["shape"] for r in ctx.last_pass_launches() if r["fp32"]] == [1]
    ctx.close()
    assert np.sqrt(np.mean((Jm / J - 1.0) ** 2)) < 3.5e-7
