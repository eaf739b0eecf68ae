"""Float64 bins cut into shares, against a plain NumPy contraction: grids of one and
two bins, so that a few hundred rows are dense enough to be staged, and row numbers
on both sides of the first share's end (512), of a second one's, and of many.

Tolerance as for the block scales: 128 units of 2^-53 of the largest sample of a
query's block (a derivative per cell spacing)."""
import numpy as np
import pytest

import test_gpu_fx as fx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("n", [511, 512, 513, 1024, 1025, 20_000])
@pytest.mark.parametrize("where", ["cell", "even", "steep"])
@pytest.mark.parametrize("shape", [(11, 11, 11), (19, 11, 9), (7, 7, 7, 7), (11, 7, 6, 7)])
def test_shares_of_staged_float64_bins(shape, where, n):
    from arbinterp_gb300 import quadcubic, tricubic
    d = len(shape)
    rng = np.random.default_rng(n)
    h = [0.1, 1 / 3, 0.0625, 0.7][:d]
    axes = [-0.4 + s * np.arange(m) for s, m in zip(h, shape)]
    V = fx._samples("steep" if where == "steep" else "smooth", axes, rng)
    G = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    pts = [g.reshape(-1) for g in G]
    lo = np.array([a[1] for a in axes])
    hi = np.array([a[-2] for a in axes])
    if where == "cell":                                  # every row in one cell
        q = lo + np.array(h) * (1.0 + 0.01 + 0.98 * rng.random((n, d)))
    else:
        q = lo + (hi - lo) * (1e-9 + (1 - 2e-9) * rng.random((n, d)))
    hh = np.array([abs(a[0] - a[1]) for a in axes])
    cls, kw = (tricubic if d == 3 else quadcubic), dict(strategy="otf", sort_threshold=0)
    o = cls(np.stack(pts + [V.reshape(-1)], 1), "quiet", **kw)
    val, grad = o.Query(q.copy())
    flat, want, slope, top = fx._reference(axes, V, q)
    assert np.array_equal(o.queryInds, flat)
    fx._compare(val[:, 0], want, top)
    fx._compare(grad * hh, slope, top[:, None])
    B = [V, fx._samples("linear", axes, rng), 1e6 * V]
    both = cls(np.stack(pts + [b.reshape(-1) for b in B], 1), "quiet", mode="both", **kw).Query(q.copy())
    for f in range(3):
        _, want, _, top = fx._reference(axes, B[f], q)
        fx._compare(both[0][:, f], want, top)
    N = np.sqrt((B[0] * B[0] + B[1] * B[1]) + B[2] * B[2])
    _, want, slope, top = fx._reference(axes, N, q)
    fx._compare(both[1][:, 0], want, top)
    fx._compare(both[2] * hh, slope, top[:, None])
