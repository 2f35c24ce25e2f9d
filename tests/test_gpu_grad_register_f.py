"""The register gradient kernels of the classes that mix f shells with p and d
shells, against the program kernel's gradient pass, as in
test_gpu_grad_register.py.

Bound: both sides keep the same primitive quartets and sum the same FP64 terms in
another order; 1e-11 of the largest element covers ~1e5 roundings of 1.1e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C1, C3 = [(0.8, 1.0)], [(6.0, 0.2), (1.3, 0.5), (0.3, 0.6)]
MIXED_F = {(0, 0, 3, 1), (0, 0, 3, 2), (1, 0, 3, 0), (1, 0, 3, 1), (1, 1, 3, 0), (2, 0, 3, 0)}


@pytest.mark.parametrize("ls", [(0, 1, 3), (0, 2, 3), (0, 1, 2, 3)])
@pytest.mark.parametrize("depth", ["one", "many"])
def test_register_gradients_with_f_vs_program_kernel(lgx, monkeypatch, ls, depth):
    pos = [[0.0, 0.0, 0.0], [1.1, -0.4, 0.7], [-0.8, 1.6, 0.3]]
    prim = {"one": [C1, C1], "many": [C3, C1]}[depth]
    shells, atoms = [], []
    for a, o in enumerate(pos):
        for l in ls:
            shells.append(lgx.Shell(l, prim[(a + l) % 2], o, pure=l > 1))
            atoms.append(a)
    bs = lgx.BasisSet(shells)
    bs.atom_of_shell = atoms
    rng = np.random.default_rng(2)
    A = rng.uniform(-1.0, 1.0, (bs.nbf, bs.nbf))
    D = A + A.T
    res = []
    for off in ("0", "1"):
        monkeypatch.setenv("LGX_DISABLE_RK", off)
        ctx = lgx.Context(0)
        ctx.set_basis(bs)
        gJ, gK, st = ctx.jk_grad(D, len(pos), 0.0)
        kernels = {r["class"]: r["kernel"] for r in ctx.last_pass_launches()}
        ctx.close()
        res.append((gJ, gK, st.prim_quartets, kernels))
    (gJ, gK, n, kernels), (rJ, rK, rn, rkernels) = res
    assert all((k == "register") == (sum(c) <= 5) for c, k in kernels.items())
    assert "register" not in rkernels.values()
    assert len(ls) < 4 or MIXED_F <= set(kernels)
    assert n == rn
    assert np.max(np.abs(gJ - rJ)) < 1e-11 * np.max(np.abs(rJ))
    assert np.max(np.abs(gK - rK)) < 1e-11 * np.max(np.abs(rK))
