"""The double-float Boys argument of the mixed scheme's J/K kernels
(ds_boys_arg_jk in libint_gb300/csrc/lgx_device.cuh), restated step by step in
numpy float32 with the FMA emulated in float64 (the product of two float32
values is exact there), against the argument in extended precision.

Bound: the argument keeps 2^-44 relative besides the 2^-48 |P| of the records
(each difference of two coordinates up to 70 then moves by 2^-47 70 = 5e-13, T by
2 sqrt(rho T) times sqrt(3) of it), so that F_m moves by less than 1e-9 (FP32
half-ulp: 6e-8)."""
import numpy as np

f32, f64 = np.float32, np.float64


def _fma(a, b, c):
    return (f64(a) * f64(b) + f64(c)).astype(f32)


def _two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def _split(x):
    h = x.astype(f32)
    return h, (x - h.astype(f64)).astype(f32)


def test_double_float_boys_argument_of_the_jk_kernels():
    rng = np.random.default_rng(1)
    n = 100000
    zb = np.exp(rng.uniform(np.log(0.05), np.log(3e4), n))
    zk = np.exp(rng.uniform(np.log(0.05), np.log(3e4), n))
    Pb = rng.uniform(-30.0, 30.0, (n, 3))
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    d = np.exp(rng.uniform(np.log(1e-4), np.log(40.0), n))
    Pk = Pb + d[:, None] * u
    (bh, bl), (kh, kl) = _split(zb), _split(zk)
    rs = (1.0 / np.sqrt((bh + kh).astype(f64))).astype(f32)
    oog = rs * rs
    rho0 = bh * kh * oog
    # residual of rho0
    p = bh * kh
    a, al = _two_sum(bh, kh)
    q = rho0 * a
    t = _fma(-rho0, al + (bl + kl), _fma(bh, kl, bl * kh))
    r = (p - q) + ((_fma(bh, kh, -p) - _fma(rho0, a, -q)) + t)
    c = r * oog
    # |P - Q|^2
    hs, lo = [], f32(0)
    for x in range(3):
        (ph, pl), (qh, ql) = _split(Pb[:, x]), _split(Pk[:, x])
        h, e = _two_sum(ph, -qh)
        l = e + (pl - ql)
        s = h * h
        lo = lo + _fma(h, h, -s)
        lo = _fma(l, _fma(f32(2), h, l), lo)
        hs.append(s)
    s1, e1 = _two_sum(hs[0], hs[1])
    s2, e2 = _two_sum(s1, hs[2])
    lo = lo + (e1 + e2)
    th = rho0 * s2
    tl = _fma(rho0, lo, _fma(c, s2, _fma(rho0, s2, -th)))
    T = th.astype(f64) + tl.astype(f64)
    L = np.longdouble
    Tref = (zb.astype(L) * zk.astype(L) / (zb.astype(L) + zk.astype(L))
            * ((Pb.astype(L) - Pk.astype(L)) ** 2).sum(1))
    rel = np.abs((T - Tref) / Tref).astype(f64)
    Tr = Tref.astype(f64)
    assert np.median(rel) < 1e-12
    rho = zb * zk / (zb + zk)
    assert np.all(rel * Tr <= 2.0 ** -44 * Tr + 2 * np.sqrt(3 * rho * Tr) * 5e-13 + rho * 1e-24)
    dF = Tr * rel * np.minimum(1.0, 6.5 / np.maximum(Tr, 1e-300))
    assert dF.max() < 1e-9
