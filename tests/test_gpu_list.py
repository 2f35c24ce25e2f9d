"""Explicit quartet lists classified on the GPU (8192 quartets and more)
against the same quartets in short lists, which the host classifies: every
class, both orders of every pair and of bra and ket, contraction depths from 1
to 1296 primitive quartets, scattered output offsets.

Bound: FP64 sets may be summed over lanes in another order (at most 1296 terms
of one sign pattern): 1e-12 of the largest value.  An FP32 set takes the same
number of lanes where the mean depth of its class is the same, and is then equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _basis(lgx):
    rng = np.random.default_rng(2)
    shells = []
    for l, n in [(0, 6), (1, 3), (0, 1), (2, 1), (1, 1), (3, 1), (0, 3), (2, 2)]:
        ex = np.exp(rng.uniform(np.log(0.2), np.log(8.0), n))
        shells.append(lgx.Shell(l, list(zip(ex, rng.uniform(0.2, 1.0, n))),
                                rng.uniform(-1.5, 1.5, 3), pure=l > 1))
    return lgx.BasisSet(shells)


@pytest.mark.parametrize("n", [8192, 8193, 20011])
@pytest.mark.parametrize("deriv", [0, 1])
def test_device_classified_list(lgx, n, deriv):
    bs = _basis(lgx)
    rng = np.random.default_rng(n + deriv)
    q = rng.integers(0, len(bs), (n, 4)).astype(np.int32)
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    out, offs, null = ctx.compute_batch(q, deriv)
    want = np.zeros_like(out)
    wnull = np.zeros_like(null)
    for k in range(0, n, 8000):
        o, f, z = ctx.compute_batch(q[k:k + 8000], deriv)
        want[offs[k]:offs[k] + o.size] = o
        wnull[k:k + 8000] = z
    assert np.array_equal(null, wnull)
    assert np.max(np.abs(out - want)) < 1e-12 * np.max(np.abs(want))
    ctx.close()


@pytest.mark.parametrize("mode", [1, 2])
def test_device_classified_mixed_list(lgx, mode):
    # one quartet more takes the list from the host's to the GPU's classification
    bs = _basis(lgx)
    q = np.random.default_rng(8).integers(0, len(bs), (8192, 4)).astype(np.int32)
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    out, offs, null = ctx.compute_batch(q, 0, mode, 0.1)
    want, _, wnull = ctx.compute_batch(q[:8191], 0, mode, 0.1)
    assert np.array_equal(null[:8191], wnull)
    assert np.max(np.abs(out[:want.size] - want)) < 1e-12 * np.max(np.abs(want))
    ctx.close()


def test_device_list_scattered_offsets_and_errors(lgx):
    torch = pytest.importorskip("torch")
    bs = _basis(lgx)
    n = 9001
    q = np.random.default_rng(5).integers(0, len(bs), (n, 4)).astype(np.int32)
    ctx = lgx.Context(0)
    ctx.set_basis(bs)
    want, offs, _ = ctx.compute_batch(q)
    # sets in reverse order, one double apart (the last quartet of the list first)
    size = np.diff(np.concatenate([offs, [want.size]]))
    rev = np.zeros(n, np.int64)
    rev[::-1] = np.concatenate([[0], np.cumsum(size[::-1] + 1)[:-1]])
    cap = int(size.sum() + n)
    d = torch.full((cap,), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.compute_batch_device(q, d.data_ptr(), cap, offsets=rev)
    got = d.cpu().numpy()
    for i in range(n):
        assert np.array_equal(got[rev[i]:rev[i] + size[i]], want[offs[i]:offs[i] + size[i]]), i
    with pytest.raises(lgx.LgxError) as e:
        ctx.compute_batch_device(q, d.data_ptr(), cap - 2, offsets=rev)
    assert e.value.status == lgx._lgx.LGX_ERR_TOO_LARGE
    for bad in (-1, len(bs)):
        qb = q.copy()
        qb[n - 1, 2] = bad
        with pytest.raises(lgx.LgxError) as e:
            ctx.compute_batch_device(qb, d.data_ptr(), cap, offsets=rev)
        assert e.value.status == lgx._lgx.LGX_ERR_INVALID_ARG
    ctx.close()
