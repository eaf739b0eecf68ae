"""Float64 fields with a component that is zero around a query: the cell's corners
give no scale, and the block is evaluated as zero unless it holds another sample.
Isolated samples put cells with zero corners and something, or nothing, in the rest
of their block beside each other.

Tolerance as for the block scales: 128 units of 2^-53 of the block's largest sample
(a derivative per cell spacing)."""
import numpy as np
import pytest

import test_gpu_fx as fx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("path", ["plain", "sparse", "dense"])
@pytest.mark.parametrize("size", [1.0, 1e-305, 3e290])
@pytest.mark.parametrize("shape", [(21, 20, 12), (9, 8, 7, 7)])
def test_isolated_samples(shape, size, path):
    from arbinterp_gb300 import quadcubic, tricubic
    d = len(shape)
    rng = np.random.default_rng(d)
    h = [0.1, 1 / 3, 0.0625, 0.7][:d]
    axes = [-0.4 + s * np.arange(n) for s, n in zip(h, shape)]
    lone = np.zeros(shape[::-1])
    lone.reshape(-1)[rng.integers(0, lone.size, lone.size // 60)] = size
    planar = np.where(np.indices(lone.shape)[0] < 5, 0.0, -0.0)
    # the steep component makes every bin uneven, so that staged queries set their own scale too
    B = [lone, planar, 1e-3 * size * fx._samples("steep", axes, rng)]
    G = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    pts = [g.reshape(-1) for g in G]
    lo = np.array([a[1] for a in axes])
    hi = np.array([a[-2] for a in axes])
    edge = 8 if d == 3 else 4
    bins = int(np.prod([(n - 3 + edge - 1) // edge for n in shape]))
    n = {"plain": 900, "sparse": 20 * bins, "dense": 150 * bins}[path]
    q = lo + (hi - lo) * (1e-9 + (1 - 2e-9) * rng.random((n, d)))
    cls, kw = (tricubic if d == 3 else quadcubic), dict(strategy="otf", sort_threshold=1 << 40 if path == "plain" else 0)
    comps = cls(np.stack(pts + [b.reshape(-1) for b in B], 1), "quiet", mode="vector", **kw).Query(q.copy())
    for f in range(3):
        _, val, _, top = fx._reference(axes, B[f], q)
        fx._compare(comps[:, f], val, top)
    val, grad = cls(np.stack(pts + [lone.reshape(-1)], 1), "quiet", **kw).Query(q.copy())
    _, want, slope, top = fx._reference(axes, lone, q)
    fx._compare(val[:, 0], want, top)
    fx._compare(grad * np.array([abs(a[0] - a[1]) for a in axes]), slope, top[:, None])
