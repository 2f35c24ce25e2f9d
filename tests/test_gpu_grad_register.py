"""The register-resident gradient kernels against the program kernel's gradient
pass (which test_gpu_jk.py holds to the oracle and to finite differences), over
bases that hold one class pattern each: pure s and p shells, HRR on either side
(p and d with s), f with s, one and many primitives (one to several lanes per
quartet), an atom with two shells.

Bound: both sides keep the same primitive quartets and sum the same FP64 terms
in another order; 1e-11 of the largest element covers ~1e5 roundings of
1.1e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C1, C3 = [(0.8, 1.0)], [(6.0, 0.2), (1.3, 0.5), (0.3, 0.6)]


@pytest.mark.parametrize("ls", [(0,), (1,), (0, 1), (0, 2), (0, 3), (0, 1, 2)])
@pytest.mark.parametrize("depth", ["one", "many"])
def test_register_gradients_vs_program_kernel(lgx, monkeypatch, ls, depth):
    pos = [[0.0, 0.0, 0.0], [1.1, -0.4, 0.7], [-0.8, 1.6, 0.3], [9.0, 4.0, -7.0]]
    prim = {"one": [C1, C1], "many": [C3, C1]}[depth]
    shells, atoms = [], []
    for a, o in enumerate(pos):
        for l in ls:
            shells.append(lgx.Shell(l, prim[(a + l) % 2], o, pure=l > 1))
            atoms.append(a)
    bs = lgx.BasisSet(shells)
    bs.atom_of_shell = atoms
    rng = np.random.default_rng(1)
    A = rng.uniform(-1.0, 1.0, (bs.nbf, bs.nbf))
    D = A + A.T
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    gJ, gK, st = ctx.jk_grad(D, len(pos), 0.0)
    low = [r for r in ctx.last_pass_launches() if sum(r["class"]) <= 4]
    assert low and all(r["kernel"] == "register" for r in low)
    ctx.close()
    monkeypatch.setenv("LGX_DISABLE_RK", "1")
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    rJ, rK, rst = ctx.jk_grad(D, len(pos), 0.0)
    assert all(r["kernel"] != "register" for r in ctx.last_pass_launches())
    ctx.close()
    assert st.prim_quartets == rst.prim_quartets
    assert np.max(np.abs(gJ - rJ)) < 1e-11 * np.max(np.abs(rJ))
    assert np.max(np.abs(gK - rK)) < 1e-11 * np.max(np.abs(rK))


@pytest.mark.parametrize("n", [150, 3000, 9000])
def test_register_derivative_sets_vs_program_kernel(lgx, monkeypatch, n):
    # every order of shells up to f; block, host- and GPU-classified list sizes
    rng = np.random.default_rng(7)
    shells = []
    for l, k in [(0, 5), (1, 3), (2, 1), (0, 1), (3, 1), (1, 1), (2, 2), (3, 2)]:
        ex = np.exp(rng.uniform(np.log(0.2), np.log(8.0), k))
        shells.append(lgx.Shell(l, list(zip(ex, rng.uniform(0.2, 1.0, k))),
                                rng.uniform(-1.5, 1.5, 3), pure=l > 1))
    bs = lgx.BasisSet(shells)
    q = rng.integers(0, len(bs), (n, 4)).astype(np.int32)
    res = []
    for off in ("0", "1"):
        monkeypatch.setenv("LGX_DISABLE_RK", off)
        ctx = lgx.Context(0)
        ctx.set_basis(bs)
        res.append(ctx.compute_batch(q, 1))
        ctx.close()
    (a, _, na), (b, _, nb) = res
    assert np.array_equal(na, nb)
    assert np.max(np.abs(a - b)) < 1e-11 * np.max(np.abs(b))
