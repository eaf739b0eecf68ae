"""Rows that need no evaluation (outside, NaN) are
recorded from the end of the workspace by the counting pass: none of them, some,
runs of whole warps, and all of them, against the row kernels (same cell
indices, values within 128 units of the largest sample, 2^-53 or 2^-24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("share", [0.0, 0.01, 0.5, 1.0])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dim", [3, 4])
def test_special_rows(dim, precision, share):
    import torch
    from arbinterp_gb300 import quadcubic, tricubic
    rng = np.random.default_rng(8)
    ax = [np.arange(n) * 0.5 - 2 for n in (12, 13, 11, 9)[:dim]]
    pts = np.stack([m.T.reshape(-1) for m in np.meshgrid(*ax, indexing="ij")], 1)
    field = np.concatenate([pts, rng.standard_normal((len(pts), 1))], 1)
    cls = tricubic if dim == 3 else quadcubic
    n = 70_001
    lo, hi = np.array([a[1] for a in ax]), np.array([a[-2] for a in ax])
    q = lo + (hi - lo) * rng.random((n, dim))
    bad = rng.random(n) < share
    if share == 0.5:
        bad = np.arange(n) // 64 % 2 == 0
    bad[100] = False
    q[bad, rng.integers(0, dim, bad.sum())] = np.where(np.arange(bad.sum()) % 3 == 0, np.nan, 99.0)
    q[100] = lo                                 # zero offset on every axis
    out = []
    for thr in (1, 1 << 30):
        ip = cls(field, "quiet", precision=precision, strategy="otf", sort_threshold=thr)
        qt = torch.from_numpy(q.copy()).cuda()
        r = ip.rQuery(qt)
        out.append([v.cpu().numpy().reshape(n, -1) for v in (r if isinstance(r, tuple) else (r,))] +
                   [ip.queryInds, qt.cpu().numpy()])
    tol = 128 * (2.0 ** -53 if precision == "fp64" else 2.0 ** -24) * np.abs(field[:, -1]).max() * 2
    for a, b in zip(out[0][:-2], out[1][:-2]):
        np.testing.assert_allclose(a, b, rtol=0, atol=tol)
        assert np.isnan(a[bad]).all()
    assert (out[0][-2] == out[1][-2]).all()
    assert np.array_equal(out[0][-1], out[1][-1], equal_nan=True)
