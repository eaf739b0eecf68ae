"""Float64 queries in block fixed point: the gathered, bin-ordered and
bin-staged evaluators against a plain NumPy contraction, on fields that stress
the block scale (steep, tiny, huge, zero, NaN and infinite samples) and on grid
edges.

Tolerance: a float64 evaluation of these sums is off by up to 60 units of 2^-53
of the largest sample of its 4^dim block (measured against quadruple
precision), the fixed-point one by up to 4; 128 such units cover both sides.
Derivatives are compared per cell spacing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ULP = 128 * 2.0 ** -53


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _weights(t):
    w = np.stack([t * (-0.5 + t * (1 - 0.5 * t)), 1 + t * t * (-2.5 + 1.5 * t), t * (0.5 + t * (2 - 1.5 * t)),
                  t * t * (-0.5 + 0.5 * t)], -1)
    d = np.stack([-0.5 + t * (2 - 1.5 * t), t * (-5 + 4.5 * t), 0.5 + t * (4 - 4.5 * t), t * (-1 + 1.5 * t)], -1)
    return w, d


def _reference(axes, V, q):
    """Flat cell indices, values, derivatives (per cell), block maxima of the grid V[(t,) z, y, x] at q."""
    d = len(axes)
    n = [len(a) for a in axes]
    base = np.zeros(len(q), dtype=np.int64)
    flat = np.zeros(len(q), dtype=np.int64)
    offs, st, cs, ws, ds, ts = np.zeros(1, dtype=np.int64), 1, 1, [], [], []
    for a in range(d):
        iu = (q[:, a] - axes[a][1]) / abs(axes[a][0] - axes[a][1])
        k = np.floor(iu)
        w, dw = _weights(iu - k)
        ws.append(w)
        ds.append(dw)
        ts.append(iu - k)
        base += k.astype(np.int64) * st
        flat += k.astype(np.int64) * cs
        offs = (np.arange(4)[:, None] * st + offs[None]).reshape(-1)
        st *= n[a]
        cs *= n[a] - 3
    blk = V.reshape(-1)[base[:, None] + offs[None]].reshape(-1, *([4] * d))

    def con(b, w):
        for u in w:
            b = (b * u.reshape(len(u), *([1] * (b.ndim - 2)), u.shape[1])).sum(-1)
        return b
    val = con(blk, ws)
    grad = np.stack([con(blk, [ds[b] if b == a else ws[b] for b in range(d)]) for a in range(d)], 1)
    if d == 4:
        S = blk
        for a in range(4):
            S = 0.5 * (np.take(S, [2, 3], -1 - a) - np.take(S, [0, 1], -1 - a))
        S = S.reshape(len(q), 16)
        T = np.concatenate([-S[:, :1], S[:, :-1] - S[:, 1:]], 1).reshape(-1, 2, 2, 2, 2)
        hb = [np.stack([t * (1 - t) ** 2, t * t * (t - 1)], -1) for t in ts]
        db = [np.stack([1 - 4 * t + 3 * t * t, 3 * t * t - 2 * t], -1) for t in ts]
        val = val + con(T, hb)
        grad = grad + np.stack([con(T, [db[b] if b == a else hb[b] for b in range(4)]) for a in range(4)], 1)
    return flat, val, grad, np.abs(blk).reshape(len(q), -1).max(1)


def _samples(kind, axes, rng):
    G = np.meshgrid(*axes[::-1], indexing="ij")[::-1]      # (x, y, z[, t]) grids, x fastest
    h = [a[1] - a[0] for a in axes]
    cells = [(g - a[0]) / s for g, a, s in zip(G, axes, h)]
    smooth = np.sin(0.31 * cells[0]) * np.cos(0.23 * cells[1]) + 0.3 * np.sin(0.4 * cells[2])
    if len(axes) == 4:
        smooth = smooth + 0.2 * np.cos(0.7 * cells[3])
    if kind == "smooth":
        return smooth
    if kind == "linear":                                   # through zero: cells far below their bin's largest sample
        return sum(c - 0.37 * len(a) for c, a in zip(cells, axes))
    if kind == "steep":                                    # e^(-1.9 cells): every bin uneven, every block within 2^9
        return np.exp(-1.9 * cells[0]) * (2 + np.cos(cells[1]))
    if kind == "noise":                                    # samples over 40 binades: the block sets the scale
        return rng.choice([-1.0, 1.0], smooth.shape) * np.exp2(rng.uniform(-40, 0, smooth.shape))
    if kind == "huge":
        return smooth * 1e305
    if kind == "tiny":
        return smooth * 1e-300
    if kind == "zeros":                                    # zero outside a box
        return np.where((cells[0] > 9) & (cells[1] > 6), smooth, 0.0)
    if kind == "nan":
        out = smooth.copy()
        out.reshape(-1)[rng.integers(0, out.size, 5)] = np.nan
        return out
    raise AssertionError(kind)


def _compare(got, ref, scale):
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    m = np.isfinite(ref)
    err = np.abs(got[m] - ref[m])
    lim = ULP * np.broadcast_to(scale, ref.shape)[m]
    assert (err <= lim).all(), (err / np.maximum(lim, 1e-320)).max()


KINDS = ["smooth", "linear", "steep", "noise", "huge", "tiny", "zeros", "nan"]
# 8^3-cell and 4^4-cell bins with remainders, one cell past a bin, and the smallest grid
SHAPES = [(21, 20, 12), (11, 12, 27), (4, 4, 5), (13, 9, 8, 7), (4, 5, 4, 4)]


# rows: gathered in query order, in bin order below and above the density at which bins are staged
@pytest.mark.parametrize("path", ["plain", "sparse", "dense"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_scalar_block_scales(kind, shape, path):
    from arbinterp_gb300 import quadcubic, tricubic
    rng = np.random.default_rng(len(shape) * 100 + shape[0])
    h = [0.1, 1 / 3, 0.0625, 0.7][: len(shape)]
    axes = [-0.4 + s * np.arange(n) for s, n in zip(h, shape)]
    V = _samples(kind, axes, rng)
    G = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    rows = np.stack([g.reshape(-1) for g in G] + [V.reshape(-1)], 1)
    edge = 8 if len(shape) == 3 else 4
    bins = int(np.prod([(n - 3 + edge - 1) // edge for n in shape]))
    nq = {"plain": 700, "sparse": 5 * bins + 3, "dense": min(150 * bins + 77, 40_000)}[path]
    lo = np.array([a[1] for a in axes])
    hi = np.array([a[-2] for a in axes])
    q = lo + (hi - lo) * rng.random((nq, len(shape)))
    q[: nq // 5] = lo + np.floor((q[: nq // 5] - lo) / (hi - lo) * (np.array(shape) - 3)) * np.array(h)   # on cell faces
    q = np.clip(q, lo, np.nextafter(hi - 1e-9 * np.array(h), -np.inf))
    flat, val, grad, top = _reference(axes, V, q)
    cls = tricubic if len(shape) == 3 else quadcubic
    o = cls(rows, "quiet", strategy="otf", sort_threshold=1 << 40 if path == "plain" else 0)
    n, g = o.Query(q.copy())
    assert np.array_equal(o.queryInds, flat)
    _compare(n[:, 0], val, top)
    hh = np.array([abs(a[0] - a[1]) for a in axes])
    _compare(g * hh, grad, top[:, None])


@pytest.mark.parametrize("path", ["plain", "sparse", "dense"])
@pytest.mark.parametrize("mode", ["vector", "both"])
@pytest.mark.parametrize("shape", [(21, 20, 12), (9, 8, 7, 7)])
def test_vector_block_scales(shape, mode, path):
    """Fields of unlike scales (one zero, one steep) side by side: each has its own."""
    from arbinterp_gb300 import quadcubic, tricubic
    rng = np.random.default_rng(5)
    h = [0.1, 1 / 3, 0.0625, 0.7][: len(shape)]
    axes = [-0.4 + s * np.arange(n) for s, n in zip(h, shape)]
    B = [1e8 * _samples("smooth", axes, rng), np.zeros(shape[::-1]), _samples("steep", axes, rng)]
    G = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    rows = np.stack([g.reshape(-1) for g in G] + [b.reshape(-1) for b in B], 1)
    edge = 8 if len(shape) == 3 else 4
    bins = int(np.prod([(n - 3 + edge - 1) // edge for n in shape]))
    nq = {"plain": 600, "sparse": 5 * bins + 3, "dense": 150 * bins + 77}[path]
    lo = np.array([a[1] for a in axes])
    hi = np.array([a[-2] for a in axes])
    q = lo + (hi - lo) * (1e-12 + (1 - 2e-9) * rng.random((nq, len(shape))))
    cls = tricubic if len(shape) == 3 else quadcubic
    o = cls(rows, "quiet", mode=mode, strategy="otf", sort_threshold=1 << 40 if path == "plain" else 0)
    res = o.Query(q.copy())
    comps = res if mode == "vector" else res[0]
    for f in range(3):
        flat, val, _, top = _reference(axes, B[f], q)
        _compare(comps[:, f], val, top)
    assert np.array_equal(o.queryInds, flat)
    if mode == "both":
        N = np.sqrt((B[0] * B[0] + B[1] * B[1]) + B[2] * B[2])
        _, val, grad, top = _reference(axes, N, q)
        _compare(res[1][:, 0], val, top)
        _compare(res[2] * np.array([abs(a[0] - a[1]) for a in axes]), grad, top[:, None])


@pytest.mark.parametrize("h", [0.1, 1 / 3, 3e-5, 7e11, 2.0 ** -20])
def test_cell_step_is_the_float64_quotient(h):
    """Points on, just below and just above cell faces: index and value as the float64 floor and fraction give them."""
    from arbinterp_gb300 import tricubic
    n = (300, 5, 5)
    axes = [h * (np.arange(n[0]) - 17.0), np.arange(5.0), np.arange(5.0)]
    G = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    V = np.cos(0.2 * G[0] / h) + G[1] + G[2]
    rows = np.stack([g.reshape(-1) for g in G] + [V.reshape(-1)], 1)
    x = axes[0][1:-3]
    x = np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x[1:], -np.inf), x[1:] - 1e-14 * h])
    q = np.stack([x, np.full(len(x), 1.5), np.full(len(x), 1.25)], 1)
    flat, val, _, top = _reference(axes, V, q)
    for threshold in (1 << 40, 0):
        o = tricubic(rows, "quiet", strategy="otf", sort_threshold=threshold)
        v, _ = o.Query(q.copy())
        assert np.array_equal(o.queryInds, flat)
        _compare(v[:, 0], val, top)
