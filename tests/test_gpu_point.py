"""A NumPy point takes one launch that leaves its results in pinned memory; the
same point as a tensor takes the row path.  Both must agree in every mode,
inside, on faces and at NaN.

Tolerance: either side is within 64 units (2^-53, mixed 2^-24) of the largest
sample of its block (per cell spacing for derivatives), so 128 cover both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _outcome(ip, q):
    """Result parts and cell index, or the error that the call raises."""
    try:
        r = ip.sQuery(q)
    except IndexError:
        return None, None
    return _parts(r), ip.queryInd


def _parts(r):
    return [np.asarray(v.cpu() if hasattr(v, "cpu") else v, dtype=np.float64).reshape(-1)
            for v in (r if isinstance(r, tuple) else (r,))]


@pytest.mark.parametrize("dim,mode", [(3, "vector"), (3, "norm"), (3, "both"), (3, "scalar"),
                                      (4, "vector"), (4, "scalar")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("eval_mode", ["otf", "table"])
def test_point_matches_rows(dim, mode, precision, eval_mode):
    import torch
    from arbinterp_gb300 import quadcubic, tricubic
    rng = np.random.default_rng(3)
    ax = [np.arange(n) * 0.25 - 1 for n in (6, 7, 9, 5)[:dim]]
    pts = np.stack([m.T.reshape(-1) for m in np.meshgrid(*ax, indexing="ij")], 1)
    field = np.concatenate([pts, rng.standard_normal((len(pts), 1 if mode == "scalar" else 3))], 1)
    cls = tricubic if dim == 3 else quadcubic
    ip = cls(field, "quiet", mode=mode, precision=precision, strategy=eval_mode)
    lo, hi = np.array([a[1] for a in ax]), np.array([a[-2] for a in ax])
    qs = list(lo + (hi - lo) * rng.random((12, dim)))
    qs += [lo, np.nextafter(hi, lo), np.where(np.arange(dim) == 1, np.nan, lo + 0.1)]
    tol = 128 * (2.0 ** -53 if precision == "fp64" else 2.0 ** -24) * np.abs(field[:, dim:]).max() * 4 * 2
    for q in qs:
        (got, gi), (want, wi) = _outcome(ip, q), _outcome(ip, torch.from_numpy(np.array(q)))
        assert gi == wi
        if got is None:                   # one rounding below an upper corner: the cell above the last
            continue
        for a, b in zip(got, want):
            assert a.shape == b.shape
            np.testing.assert_allclose(a, b, rtol=0, atol=tol)
    assert ip.sQuery(hi + 0.1) is np.nan
    with pytest.raises(IndexError):       # the cell above the last
        ip.sQuery(hi)
    with pytest.raises(IndexError):
        ip.sQuery(torch.from_numpy(hi))
