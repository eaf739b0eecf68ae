"""Float64 queries on grid points: the sample itself and central differences, bit for
bit as float64 arithmetic gives them, whatever the samples around are, on the row,
bin-ordered and staged paths.

The derivative of float64 arithmetic there is (f(+1) / 2 - f(-1) / 2) times 1 / h, each
operation rounded once (halves are exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = 0.25                                     # exact quotients: every fraction of a node is zero


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _field(kind, shape, rng):
    """Samples [x, y, z(, t)]."""
    G = np.meshgrid(*[np.arange(n, dtype=float) for n in shape], indexing="ij")
    smooth = np.sin(0.31 * G[0]) * np.cos(0.23 * G[1]) + 0.3 * np.sin(0.4 * G[2])
    return {"smooth": smooth, "linear": sum(g - 0.37 * n for g, n in zip(G, shape)),
            "steep": np.exp(-1.9 * G[0]) * (2 + np.cos(G[1])),
            "binades": rng.choice([-1.0, 1.0], smooth.shape) * np.exp2(rng.uniform(-40, 0, smooth.shape)),
            "tiny": smooth * 1e-300}[kind]


def _nodes(shape, n, rng):
    """n rows of node indices inside the volume, below the upper faces."""
    return np.stack([rng.integers(1, m - 2, n) for m in shape], 1)


def _slopes(V, k):
    out = []
    for a in range(V.ndim):
        e = np.zeros(V.ndim, dtype=int)
        e[a] = 1
        out.append((0.5 * V[tuple((k + e).T)] - 0.5 * V[tuple((k - e).T)]) * (1 / H))
    return np.stack(out, 1)


@pytest.mark.parametrize("path", ["plain", "sparse", "dense"])
@pytest.mark.parametrize("shape", [(21, 12, 13), (9, 8, 7, 7)])
@pytest.mark.parametrize("kind", ["smooth", "linear", "steep", "binades", "tiny"])
def test_grid_points_return_their_samples(kind, shape, path):
    from arbinterp_gb300 import quadcubic, tricubic
    rng = np.random.default_rng(len(shape))
    d = len(shape)
    edge = 8 if d == 3 else 4
    bins = int(np.prod([(n - 3 + edge - 1) // edge for n in shape]))
    n = {"plain": 500, "sparse": 20 * bins, "dense": 150 * bins}[path]
    cls, kw = (tricubic if d == 3 else quadcubic), dict(strategy="otf", sort_threshold=1 << 40 if path == "plain" else 0)
    G = np.meshgrid(*[H * (np.arange(m) - 1.0) for m in shape], indexing="ij")
    k = _nodes(shape, n, rng)
    q = H * (k - 1.0)
    q[::3] += H * rng.random((len(q[::3]), d))           # other queries beside them in a warp
    at = np.arange(n) % 3 != 0
    V = _field(kind, shape, rng)
    rows = np.stack([g.reshape(-1) for g in G] + [V.reshape(-1)], 1)
    val, grad = cls(rows, "quiet", **kw).Query(q.copy())
    assert np.array_equal(val[at, 0], V[tuple(k[at].T)])
    assert np.array_equal(grad[at], _slopes(V, k[at]))
    B = [_field(kind, shape, rng), np.zeros(shape), 1e3 * V]
    rows = np.stack([g.reshape(-1) for g in G] + [b.reshape(-1) for b in B], 1)
    comps = cls(rows, "quiet", mode="vector", **kw).Query(q.copy())
    o = cls(rows, "quiet", mode="both", **kw)
    both = o.Query(q.copy())
    N = o._grid64.view(*shape[::-1], 4)[..., 3].cpu().numpy().transpose(*range(d - 1, -1, -1))
    for f in range(3):
        want = B[f][tuple(k[at].T)]
        assert np.array_equal(comps[at, f], want) and np.array_equal(both[0][at, f], want)
    assert np.array_equal(both[1][at, 0], N[tuple(k[at].T)])
    assert np.array_equal(both[2][at], _slopes(N, k[at]))


def test_points_and_infinite_neighbours():
    """A point query takes the same path; 0 * inf is NaN as in the weighted sum."""
    from arbinterp_gb300 import tricubic
    shape = (8, 8, 8)
    rng = np.random.default_rng(1)
    V = _field("binades", shape, rng)
    V[5, 5, 5] = np.inf
    G = np.meshgrid(*[H * (np.arange(m) - 1.0) for m in shape], indexing="ij")
    o = tricubic(np.stack([g.reshape(-1) for g in G] + [V.reshape(-1)], 1), "quiet", strategy="otf")
    v, g = o.Query(np.array([H, 0.0, H]))
    assert v == V[2, 1, 2] and np.array_equal(g, _slopes(V, np.array([[2, 1, 2]]))[0])
    v, g = o.Query(np.array([2 * H, 2 * H, 2 * H]))
    assert np.isnan(v) and np.isnan(g).all()
