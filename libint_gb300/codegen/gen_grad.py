"""Generates the unrolled per-class code of the register-resident gradient
kernels (csrc/gen/grad_classes.cuh, grad_unit_XX.cu, grad_dispatch.cu).

The gradient pass needs no derivative integrals, only their sum with the
two-particle density G_abcd (one for J, one for K).  So the density goes
through the transposes of the solid-harmonic transform and of the HRR once per
contracted quartet, to weights W_ef over the (e0|f0) set, and every primitive
quartet contracts its VRR values with them: with
  S = sum W_ef (e|f),  V_i = sum W_ef (e+1_i|f),  U_i = sum W_ef (e|f+1_i)
(2 a = twice the exponent of the centre; both factors act on primitives)
  d/dA_i : 2a_A V_i - sum W_ef e_i (e-1_i|f) + dAB_i
  d/dB_i : 2a_B (V_i + AB_i S) - dAB_i
  d/dD_i : 2a_D (U_i + CD_i S) - dCD_i,   d/dC = -(d/dA + d/dB + d/dD),
where dAB, dCD are the derivatives of the HRR with respect to AB, CD at fixed
contracted (e0|f0) (reverse-mode: every HRR step t = s1 + AB_i s2 adds W_t s2).
Relations: VRR src/bin/libint/vrr_11_twoprep_11.h:145-223,305-383, HRR
src/bin/libint/hrr.h:246-347, translational invariance and the density factors
tests/hartree-fock/hartree-fock++.cc:1909-1973.

Per class:
  weights<T>(G, AB, CD, W): spherical density -> W (kNacc values);
  prim<T>(F, g, WJ, WK, s, I): one primitive quartet: s = {S, V, U} of J and K
      (kSums values), I += contracted (e0|f0), e from la-1;
  tail<T>(I, G, W, AB, CD, lo, dab, dcd): the terms without an exponent.

First-derivative shell sets of explicit lists (DerivCls): contracted (e0|f0)
accumulators, unweighted and weighted by 2a of A, B and D, then per centre and
direction the HRR of the raised and lowered sets (master_rrs_list.h:52-55) and
the solid-harmonic transform; centre C by translational invariance.
  prim<T>(F, g, w, I): w = 2a of A, B, D;
  sets<T>(I, AB, CD, v): v[ctr * 3 + dir][kNsph] of A, B, D.

usage: python libint_gb300/codegen/gen_grad.py
"""
from __future__ import annotations

import math
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)
from gen_rk import (RK_MAX_L_STORE, Emitter, _write_if_changed, comps, first_dir, lit, ncart,  # noqa: E402
                    rk_classes, sh, sph_matrix)

GEN_DIR = os.path.join(os.path.dirname(HERE), "csrc", "gen")
# total angular momentum of the classes (see rk_grad_kernel for where it ends)
GRAD_MAX_L = 5
# classes of the derivative store kernels (see rk_deriv_kernel)
DERIV_MAX_L = 3
N_UNITS = 8
XYZ = "xyz"


class Vrr:
    """(e|f)^(m) nodes of one class as straight-line code (as in gen_rk)."""

    def __init__(self, em):
        self.em = em
        self.names = {}
        self.used = set()

    def node(self, e, f, m):
        key = (e, f, m)
        if key in self.names:
            return self.names[key]
        if sum(e) == 0 and sum(f) == 0:
            self.names[key] = "F[%d]" % m
            return self.names[key]
        if sum(f) > 0:
            j = first_dir(f)
            f1 = sh(f, j, -1)
            expr = "fma(g.WQ%s, %s, g.QC%s * %s)" % (XYZ[j], self.node(e, f1, m + 1), XYZ[j],
                                                     self.node(e, f1, m))
            if f1[j] > 0:
                f2 = sh(f1, j, -1)
                self.used.add(("e", f1[j]))
                expr = "fma(oo2e_%d, fma(-g.roe, %s, %s), %s)" % (
                    f1[j], self.node(e, f2, m + 1), self.node(e, f2, m), expr)
            if e[j] > 0:
                self.used.add(("ze", e[j]))
                expr = "fma(oo2ze_%d, %s, %s)" % (e[j], self.node(sh(e, j, -1), f1, m + 1), expr)
        else:
            i = first_dir(e)
            e1 = sh(e, i, -1)
            expr = "fma(g.WP%s, %s, g.PA%s * %s)" % (XYZ[i], self.node(e1, f, m + 1), XYZ[i],
                                                     self.node(e1, f, m))
            if e1[i] > 0:
                e2 = sh(e1, i, -1)
                self.used.add(("z", e1[i]))
                expr = "fma(oo2z_%d, fma(-g.roz, %s, %s), %s)" % (
                    e1[i], self.node(e2, f, m + 1), self.node(e2, f, m), expr)
        self.names[key] = self.em.tmp(expr)
        return self.names[key]

    def factors(self):
        src = {"z": "oo2z", "e": "oo2e", "ze": "oo2ze"}
        return ["    const T %s_%d = T(%d) * g.%s;" % (src[k], n, n, src[k])
                for k, n in sorted(self.used)]


def gen_class(la, lb, lc, ld):
    L = la + lb + lc + ld
    es = [e for le in range(la, la + lb + 1) for e in comps(le)]
    fs = [f for lf in range(lc, lc + ld + 1) for f in comps(lf)]
    w_index = {(e, f): k for k, (e, f) in enumerate((e, f) for e in es for f in fs)}
    # contracted (e0|f0) of the tail: e from la - 1 (lowering of A)
    low = [e for e in comps(la - 1)] if la > 0 else []
    i_index = {(e, f): k for k, (e, f) in enumerate((e, f) for e in low + es for f in fs)}

    # ------------------------------------------------ transposed transforms
    ls = [la, lb, lc, ld]
    npure = [2 * l + 1 if l >= 2 else ncart(l) for l in ls]
    em = Emitter()
    cur = ["G[%d]" % i for i in range(math.prod(npure))]
    dims = list(npure)
    for k in (3, 2, 1, 0):
        if ls[k] < 2:
            continue
        M = sph_matrix(ls[k])
        nc = ncart(ls[k])
        outer, inner = math.prod(dims[:k]), math.prod(dims[k + 1:])
        nxt = []
        for oo in range(outer):
            for c in range(nc):
                for ii in range(inner):
                    terms = [(M[p][c], cur[(oo * dims[k] + p) * inner + ii])
                             for p in range(dims[k]) if M[p][c] != 0.0]
                    expr = None
                    for cf, s in terms:
                        expr = "%s * %s" % (lit(cf), s) if expr is None else \
                            "fma(%s, %s, %s)" % (lit(cf), s, expr)
                    nxt.append(em.tmp(expr))
        cur = nxt
        dims[k] = nc

    # ------------------------------------------------ HRR graph
    steps = []   # (key, direction name, s1, s2) in evaluation order
    seen = {}

    def bra(a, b, f):
        if sum(b) == 0:
            return ("i", a, f)
        key = ("b", a, b, f)
        if key not in seen:
            i = first_dir(b)
            s1 = bra(sh(a, i, 1), sh(b, i, -1), f)
            s2 = bra(a, sh(b, i, -1), f)
            seen[key] = True
            steps.append((key, "AB", i, s1, s2))
        return key

    def ket(a, b, c, d):
        if sum(d) == 0:
            return bra(a, b, c)
        key = ("k", a, b, c, d)
        if key not in seen:
            j = first_dir(d)
            s1 = ket(a, b, sh(c, j, 1), sh(d, j, -1))
            s2 = ket(a, b, c, sh(d, j, -1))
            seen[key] = True
            steps.append((key, "CD", j, s1, s2))
        return key

    outs = [ket(a, b, c, d) for a in comps(la) for b in comps(lb) for c in comps(lc)
            for d in comps(ld)]

    def reverse(em):
        """Adjoints of every node: expressions gathered over its uses."""
        adj = {}
        for o, v in zip(outs, cur):
            adj.setdefault(o, []).append((None, v))

        def close(key):
            expr = None
            for cf, v in sorted(adj[key], key=lambda t: t[0] is not None):
                if cf is None:
                    expr = v if expr is None else "%s + %s" % (expr, v)
                else:
                    expr = "%s * %s" % (cf, v) if expr is None else "fma(%s, %s, %s)" % (cf, v, expr)
            return expr if expr.replace("[", "").replace("]", "").isalnum() else em.tmp(expr)

        val = {}
        for key, vec, i, s1, s2 in reversed(steps):
            t = close(key)
            val[key] = t
            adj.setdefault(s1, []).append((None, t))
            adj.setdefault(s2, []).append(("%s[%d]" % (vec, i), t))
        for (e, f) in w_index:
            val[("i", e, f)] = close(("i", e, f))
        return val

    val = reverse(em)
    for (e, f), k in w_index.items():
        em.lines.append("    W[%d] = %s;" % (k, val[("i", e, f)]))
    weights_body = em.lines

    # ------------------------------------------------ primitive stage
    pem = Emitter()
    vrr = Vrr(pem)
    targets = []
    for le in range(max(la - 1, 0), la + lb + 2):
        for lf in range(lc, lc + ld + 2):
            if lf == lc + ld + 1 and not (la <= le <= la + lb):
                continue
            targets += [(e, f) for e in comps(le) for f in comps(lf)]
    first = set()

    def add(acc, w, v):
        # the first term of a sum is a product
        if acc in first:
            pem.lines.append("    %s = fma(%s, %s, %s);" % (acc, w, v, acc))
        else:
            first.add(acc)
            pem.lines.append("    %s = %s * %s;" % (acc, w, v))

    for e, f in targets:
        v = vrr.node(e, f, 0)
        if (e, f) in i_index:
            pem.lines.append("    I[%d] += %s;" % (i_index[(e, f)], v))
        for x, W in enumerate(("WJ", "WK")):
            o = 7 * x
            if (e, f) in w_index:
                add("s[%d]" % o, "%s[%d]" % (W, w_index[(e, f)]), v)
            for i in range(3):
                if e[i] > 0 and (sh(e, i, -1), f) in w_index:
                    add("s[%d]" % (o + 1 + i), "%s[%d]" % (W, w_index[(sh(e, i, -1), f)]), v)
                if f[i] > 0 and (e, sh(f, i, -1)) in w_index:
                    add("s[%d]" % (o + 4 + i), "%s[%d]" % (W, w_index[(e, sh(f, i, -1))]), v)
    assert len(first) == 14
    prim_body = vrr.factors() + pem.lines

    # ------------------------------------------------ tail
    tem = Emitter()
    tem.n = 100000  # apart from the names of the reverse sweep
    for i in range(3):
        tem.lines.append("    lo[%d] = T(0);" % i)
        for (e, f), k in w_index.items():
            if e[i] > 0:
                el = sh(e, i, -1)
                tem.lines.append("    lo[%d] = fma(T(%d) * W[%d], I[%d], lo[%d]);" %
                                 (i, e[i], k, i_index[(el, f)], i))
    tem.lines.append("    dab[0] = dab[1] = dab[2] = T(0);")
    tem.lines.append("    dcd[0] = dcd[1] = dcd[2] = T(0);")
    if steps:
        rem = Emitter()
        # the transposed transform again (same expressions, from G)
        rem.lines = [x for x in weights_body if " W[" not in x]
        rem.n = em.n
        tem.lines += rem.lines
        fwd = {}

        def value(key):
            if key[0] == "i":
                return "I[%d]" % i_index[(key[1], key[2])]
            return fwd[key]

        need = {s2 for _, _, _, _, s2 in steps}
        changed = True
        while changed:  # values that an exponent-free term reads, transitively
            changed = False
            for key, _, _, s1, s2 in steps:
                if key in need and not {s1, s2} <= need:
                    need |= {s1, s2}
                    changed = True
        for key, vec, i, s1, s2 in steps:
            if key in need:
                fwd[key] = tem.tmp("fma(%s[%d], %s, %s)" % (vec, i, value(s2), value(s1)))
            dst = "dab" if vec == "AB" else "dcd"
            tem.lines.append("    %s[%d] = fma(%s, %s, %s[%d]);" % (dst, i, val[key], value(s2),
                                                                    dst, i))
    tail_body = tem.lines

    key = "%d, %d, %d, %d" % (la, lb, lc, ld)
    s = ["template <>\nstruct GradCls<%s> {" % key,
         "  static constexpr int kMmax = %d, kNacc = %d, kNI = %d;" % (L + 1, len(w_index),
                                                                     len(i_index)),
         "  static constexpr int kN0 = %d, kN1 = %d, kN2 = %d, kN3 = %d;" % tuple(npure),
         "  static constexpr bool kBraHrr = %s, kKetHrr = %s, kTail = %s;" %
         tuple("true" if x else "false" for x in (lb > 0, ld > 0, la > 0 or ld > 0)),
         "  template <typename T>\n  static __device__ __forceinline__ void weights(const T* G, "
         "const T* AB, const T* CD, T* W) {"]
    s += weights_body
    s += ["  }", "  template <typename T>\n  static __device__ __forceinline__ void prim(const T* F, "
          "const Geo<T>& g, const T* WJ, const T* WK, T* s, T* I) {"]
    s += prim_body
    s += ["  }", "  template <typename T>\n  static __device__ __forceinline__ void tail(const T* I, "
          "const T* G, const T* W, const T* AB, const T* CD, T* lo, T* dab, T* dcd) {"]
    s += tail_body
    s += ["  }", "};"]
    return "\n".join(s)


def gen_deriv_class(la, lb, lc, ld):
    ls = [la, lb, lc, ld]
    acc = {}      # (weight, e, f) -> accumulator
    memo = {}
    em = Emitter()

    def leaf(w, e, f):
        k = acc.setdefault((w, e, f), len(acc))
        return "I[%d]" % k

    def bra(w, a, b, f):
        if sum(b) == 0:
            return leaf(w, a, f)
        key = (w, "b", a, b, f)
        if key not in memo:
            i = first_dir(b)
            memo[key] = em.tmp("fma(AB[%d], %s, %s)" % (i, bra(w, a, sh(b, i, -1), f),
                                                       bra(w, sh(a, i, 1), sh(b, i, -1), f)))
        return memo[key]

    def ket(w, a, b, c, d):
        if sum(d) == 0:
            return bra(w, a, b, c)
        key = (w, "k", a, b, c, d)
        if key not in memo:
            j = first_dir(d)
            memo[key] = em.tmp("fma(CD[%d], %s, %s)" % (j, ket(w, a, b, c, sh(d, j, -1)),
                                                       ket(w, a, b, sh(c, j, 1), sh(d, j, -1))))
        return memo[key]

    nsph = None
    for x, pos in enumerate((0, 1, 3)):  # A, B, D
        for i in range(3):
            vals = []
            for a in comps(la):
                for b in comps(lb):
                    for c in comps(lc):
                        for d in comps(ld):
                            q = [a, b, c, d]
                            up = list(q)
                            up[pos] = sh(q[pos], i, 1)
                            expr = ket(x + 1, *up)
                            if q[pos][i] > 0:
                                dn = list(q)
                                dn[pos] = sh(q[pos], i, -1)
                                n = q[pos][i]
                                low = ket(0, *dn)
                                expr = em.tmp("%s - %s" % (expr, low) if n == 1 else
                                              "fma(T(-%d), %s, %s)" % (n, low, expr))
                            vals.append(expr)
            dims = [ncart(l) for l in ls]
            for k in range(4):
                if ls[k] < 2:
                    continue
                M = sph_matrix(ls[k])
                npure = 2 * ls[k] + 1
                outer, inner = math.prod(dims[:k]), math.prod(dims[k + 1:])
                nxt = []
                for oo in range(outer):
                    for p in range(npure):
                        for ii in range(inner):
                            expr = None
                            for c in range(dims[k]):
                                if M[p][c] != 0.0:
                                    src = vals[(oo * dims[k] + c) * inner + ii]
                                    expr = "%s * %s" % (lit(M[p][c]), src) if expr is None else \
                                        "fma(%s, %s, %s)" % (lit(M[p][c]), src, expr)
                            nxt.append(em.tmp(expr))
                vals = nxt
                dims[k] = npure
            nsph = len(vals)
            for k, v in enumerate(vals):
                em.lines.append("    v[%d] = %s;" % ((3 * x + i) * nsph + k, v))
    sets_body = em.lines

    pem = Emitter()
    vrr = Vrr(pem)
    by = {}
    for (w, e, f), k in acc.items():
        by.setdefault((e, f), []).append((w, k))
    for e, f in sorted(by, key=lambda t: (sum(t[0]), sum(t[1]), t)):
        v = vrr.node(e, f, 0)
        for w, k in sorted(by[(e, f)]):
            if w == 0:
                pem.lines.append("    I[%d] += %s;" % (k, v))
            else:
                pem.lines.append("    I[%d] = fma(w[%d], %s, I[%d]);" % (k, w - 1, v, k))
    prim_body = vrr.factors() + pem.lines

    s = ["template <>\nstruct DerivCls<%d, %d, %d, %d> {" % (la, lb, lc, ld),
         "  static constexpr int kMmax = %d, kNacc = %d, kNsph = %d;" % (sum(ls) + 1, len(acc), nsph),
         "  static constexpr int kN0 = %d, kN1 = %d, kN2 = %d, kN3 = %d;" %
         tuple(2 * l + 1 if l >= 2 else ncart(l) for l in ls),
         "  template <typename T>\n  static __device__ __forceinline__ void prim(const T* F, "
         "const Geo<T>& g, const T* w, T* I) {"]
    s += prim_body
    s += ["  }", "  template <typename T>\n  static __device__ __forceinline__ void sets(const T* I, "
          "const T* AB, const T* CD, T* v) {"]
    s += sets_body
    s += ["  }", "};"]
    return "\n".join(s)


def main():
    os.makedirs(GEN_DIR, exist_ok=True)
    classes = rk_classes(GRAD_MAX_L)
    parts = ["// GENERATED by libint_gb300/codegen/gen_grad.py -- do not edit.",
             "// Unrolled density weights, primitive stage and tail of the",
             "// register-resident gradient kernels (see gen_grad.py).",
             "#pragma once", '#include "../lgx_rk_common.cuh"', "", "namespace lgx {",
             "namespace rk {", "", "template <int LA, int LB, int LC, int LD>", "struct GradCls;",
             "template <int LA, int LB, int LC, int LD>", "struct DerivCls;", ""]
    for c in classes:
        parts += [gen_class(*c), ""]
    for c in rk_classes(DERIV_MAX_L):
        parts += [gen_deriv_class(*c), ""]
    parts += ["}  // namespace rk", "}  // namespace lgx"]
    _write_if_changed(os.path.join(GEN_DIR, "grad_classes.cuh"), "\n".join(parts) + "\n")

    classes = sorted(classes, key=lambda c: -sum(c))
    names, decls = [], []
    items = [("grad", c) for c in classes] + [("deriv", c) for c in rk_classes(DERIV_MAX_L)]
    items += [("one0", c) for c in rk_classes(RK_MAX_L_STORE)]
    items += [("one1", c) for c in rk_classes(DERIV_MAX_L)]
    items.sort(key=lambda t: -sum(t[1]))
    for k in range(N_UNITS):
        name = "grad_unit_%02d.cu" % k
        names.append(name)
        lines = ["// GENERATED by libint_gb300/codegen/gen_grad.py -- do not edit.",
                 '#include "../lgx_rkgrad.cuh"', "", "namespace lgx {"]
        for kind, c in items[k::N_UNITS]:
            fn = "rk_%s_launch_%d%d%d%d" % ((kind,) + c)
            decls.append((kind, c, fn))
            if kind.startswith("one"):
                lines.append("cudaError_t %s(const EriArgs& a, int blocks, cudaStream_t st) {" % fn)
                lines.append("  return rk_one_launch_one<%d, %d, %d, %d, %s>(a, blocks, st);" %
                             (c + (kind[3],)))
                lines.append("}")
                continue
            lines.append("cudaError_t %s(const EriArgs& a, long long work, int nsm, "
                         "cudaStream_t st) {" % fn)
            lines.append("  return rk_%s_launch_one<%d, %d, %d, %d>(a, work, nsm, st);" %
                         ((kind,) + c))
            lines.append("}")
        lines.append("}  // namespace lgx")
        _write_if_changed(os.path.join(GEN_DIR, name), "\n".join(lines) + "\n")
    d = ["// GENERATED by libint_gb300/codegen/gen_grad.py -- do not edit.",
         "// Run-time dispatch of the register-resident derivative kernels.",
         '#include "../lgx_kernels.cuh"', "", "namespace lgx {"]
    for kind, _, fn in sorted(decls):
        d.append("cudaError_t %s(const EriArgs& a, %s, cudaStream_t st);" %
                 (fn, "int blocks" if kind.startswith("one") else "long long work, int nsm"))
    for name, lmax in (("grad", GRAD_MAX_L), ("deriv", DERIV_MAX_L)):
        d += ["", "cudaError_t rk_%s_launch(int la, int lb, int lc, int ld, const EriArgs& a, "
              "long long work, int nsm," % name, "                           cudaStream_t st) {",
              "  switch (((la * 8 + lb) * 8 + lc) * 8 + ld) {"]
        for kind, c, fn in sorted(decls):
            if kind == name:
                d.append("    case %d: return %s(a, work, nsm, st);" %
                         (((c[0] * 8 + c[1]) * 8 + c[2]) * 8 + c[3], fn))
        d += ["  }", "  return cudaErrorNotSupported;", "}", "",
              "bool rk_%s_available(int la, int lb, int lc, int ld) {" % name,
              "  return la <= 3 && lc <= 3 && la + lb + lc + ld <= %d;" % lmax, "}"]
    d += ["", "// One quartet over several blocks (derivative order 0 or 1).",
          "cudaError_t rk_one_launch(int deriv, int la, int lb, int lc, int ld, const EriArgs& a, "
          "int blocks,", "                          cudaStream_t st) {",
          "  switch ((((deriv * 8 + la) * 8 + lb) * 8 + lc) * 8 + ld) {"]
    for kind, c, fn in sorted(decls):
        if kind.startswith("one"):
            d.append("    case %d: return %s(a, blocks, st);" %
                     ((((int(kind[3]) * 8 + c[0]) * 8 + c[1]) * 8 + c[2]) * 8 + c[3], fn))
    d += ["  }", "  return cudaErrorNotSupported;", "}", "}  // namespace lgx"]
    _write_if_changed(os.path.join(GEN_DIR, "grad_dispatch.cu"), "\n".join(d) + "\n")
    return names + ["grad_dispatch.cu"]


if __name__ == "__main__":
    print("\n".join(main()))
