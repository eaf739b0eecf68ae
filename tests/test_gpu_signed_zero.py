"""A bound of the volume at zero takes coordinates of both signs of zero, as the
comparison of floats does: the same index, value and gradient for -0.0 as for
+0.0, the caller's row unchanged, on every path in both precisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = (12, 11, 10)


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rows(side, zero, axis, n=N):
    """Field rows whose volume begins (lo) or ends (hi) at `zero` along `axis`."""
    axes = []
    for a, m in enumerate(n):
        k = np.arange(m) - (1 if side == "lo" else m - 2) if a == axis else np.arange(m) + 3
        x = 0.25 * k
        x[x == 0] = zero
        axes.append(x)
    G = np.meshgrid(*axes, indexing="ij")
    val = np.cos(0.8 * G[0]) + G[1] * G[2] + sum(0.1 * g for g in G)
    return axes, np.stack([g.reshape(-1) for g in G] + [val.reshape(-1)], 1)


def _queries(axes, axis, n, value):
    rng = np.random.default_rng(3)
    lo = np.array([a[1] for a in axes])
    hi = np.array([a[-2] for a in axes])
    q = lo + (hi - lo) * (0.05 + 0.7 * rng.random((n, len(axes))))
    q[:, axis] = value
    return q


@pytest.mark.parametrize("axis", [0, 1])     # the last axis' upper face lies beyond the table: IndexError
@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("side", ["lo", "hi"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_bounds_take_both_zeros(precision, side, zero, axis):
    import torch
    from arbinterp_gb300 import tricubic
    axes, rows = _rows(side, zero, axis)
    # gathered, in bin order, and staged (two bins)
    for n, threshold in ((200, 1 << 40), (200, 0), (3000, 0)):
        o = tricubic(rows, "quiet", precision=precision, strategy="otf", sort_threshold=threshold)
        got = []
        for v in (zero, -zero):
            q = _queries(axes, axis, n, v)
            for dev in (False, True):
                qq = torch.from_numpy(q.copy()).cuda() if dev else q.copy()
                val, grad = o.Query(qq)
                after = qq.cpu().numpy() if dev else qq
                assert np.array_equal(after, q) and np.array_equal(np.signbit(after), np.signbit(q))
                val, grad = (np.asarray(t.cpu() if dev else t) for t in (val, grad))
                assert np.isfinite(val).all() and np.isfinite(grad).all()
                got.append((o.queryInds, val, grad))
        for g in got[1:]:
            for a, b in zip(got[0], g):
                assert np.array_equal(a, b)
    points = [o.Query(np.array(_queries(axes, axis, 1, v)[0])) + (o.queryInd,) for v in (zero, -zero)]
    assert np.isfinite(points[0][0]) and points[0][2] == points[1][2]
    assert points[0][0] == points[1][0] and np.array_equal(points[0][1], points[1][1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_bounds_4d(precision):
    from arbinterp_gb300 import quadcubic
    axes, rows = _rows("lo", 0.0, 0, (9, 8, 7, 7))
    for n, threshold in ((100, 1 << 40), (5000, 0)):
        o = quadcubic(rows, "quiet", precision=precision, strategy="otf", sort_threshold=threshold)
        res = [o.Query(_queries(axes, 0, n, v)) for v in (0.0, -0.0)]
        assert np.isfinite(res[0][0]).all()
        assert all(np.array_equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_bounds_adjoint_batch_and_trajectories(precision):
    import torch
    from arbinterp_gb300 import tricubic
    from arbinterp_gb300.autograd import TricubicField
    from arbinterp_gb300.batched import BatchedTricubic
    axes, rows = _rows("lo", 0.0, 0)
    n = 500
    qs = [torch.from_numpy(_queries(axes, 0, n, v)).cuda() for v in (0.0, -0.0)]
    for binned in (False, True):
        F = TricubicField(rows, precision=precision, binned_adjoint=binned)
        v = F.initial_values().requires_grad_(True)
        up = (torch.ones(n, dtype=torch.float64, device="cuda"), torch.ones(n, 3, dtype=torch.float64, device="cuda"))
        res = []
        for q in qs:
            x = q.clone().requires_grad_(True)
            res.append(torch.autograd.grad(F(v, x), (v, x), up))
        assert res[0][0].abs().sum() > 0 and torch.equal(res[0][1], res[1][1])
        # sums of at most n float32 terms in no fixed order
        assert torch.allclose(res[0][0], res[1][0], rtol=0, atol=n * 2.0 ** -24 * float(res[0][0].abs().max()))
    B = BatchedTricubic([rows, rows], precision=precision)
    q = torch.cat(qs)
    val, grad = B.query(q, [n, n])
    assert torch.isfinite(val).all() and torch.equal(val[:n], val[n:]) and torch.equal(grad[:n], grad[n:])
    o = tricubic(rows, "quiet", precision=precision)
    for q in qs:
        o.trajectories(q, torch.zeros_like(q), 0.01, 3, coef=0.0)
        assert o.lost == 0
