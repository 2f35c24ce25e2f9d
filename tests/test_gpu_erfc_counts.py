"""Primitive quartets of attenuated J/K passes: those whose integrals vanish enter
no VRR and are not counted (lgx_jk_stats.prim_quartets, and the operation counts
that are made from it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_vanishing_erfc_quartets_are_not_counted(lgx):
    # one primitive of exponent 1 on two centres 40 bohr apart: (00|00), (11|00) and
    # (11|11) pass the screens (the pair 10 does not); for (11|00) T = 1600 and, at
    # omega = 0.4, s T = 1600 * 0.16 / 1.16 = 221 > 50
    bs = lgx.BasisSet([lgx.Shell(0, [(1.0, 1.0)], [x, 0.0, 0.0], pure=False) for x in (0.0, 40.0)])
    D = np.eye(2)
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    got = {}
    for op, omega in (("coulomb", 0.0), ("erf_coulomb", 0.4), ("erfc_coulomb", 0.4)):
        ctx.set_operator(lgx.Operator[op], omega)
        J, K, st = ctx.jk(D, 0.0, 0)
        assert sum(r["prim_quartets"] for r in ctx.last_pass_launches()) == st.prim_quartets
        got[op] = J, st.prim_quartets, st.flops_fp64
    ctx.close()
    assert [got[op][1] for op in got] == [3, 3, 2]
    assert got["erfc_coulomb"][2] < got["coulomb"][2]
    # the Coulomb integrals are the sum of the two
    J = {op: got[op][0] for op in got}
    assert np.max(np.abs(J["erf_coulomb"] + J["erfc_coulomb"] - J["coulomb"])) < 1e-14
