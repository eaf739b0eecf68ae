"""A cell floor beyond 32 bits (an axis whose first spacing is tiny: the spacing is
taken from the first two values) gives an index beyond the table, whatever its
low 32 bits are: IndexError on points and rows, a lost particle, no gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = 2.0 ** -40


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rows(axis, dim=3):
    axes = [0.5 * np.arange(m) for m in (9, 8, 8, 7)[:dim]]
    axes[axis] = np.concatenate([[0.0, H], 1.0 + np.arange(len(axes[axis]) - 2)])
    G = np.meshgrid(*axes, indexing="ij")
    return axes, np.stack([g.reshape(-1) for g in G] + [sum(np.cos(g) for g in G).reshape(-1)], 1)


def _point(axes, axis, low):
    """Inside the volume, with a floor of 700 * 2^32 + low along `axis`."""
    q = np.array([a[2] + 0.125 for a in axes])
    q[axis] = H + (700 * 2.0 ** 32 + low + 0.5) * H
    return q


@pytest.mark.parametrize("low", [0, 2, -3])
@pytest.mark.parametrize("dim,axis", [(3, 0), (3, 1), (3, 2), (4, 1), (4, 3)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_floors_beyond_32_bits_stay_out_of_the_table(precision, dim, axis, low):
    import torch
    from arbinterp_gb300 import quadcubic, tricubic
    axes, rows = _rows(axis, dim)
    for threshold in (1 << 40, 0):
        o = (tricubic if dim == 3 else quadcubic)(rows, "quiet", precision=precision, strategy="otf",
                                                  sort_threshold=threshold)
        q = _point(axes, axis, low)
        assert all(float(l) <= v <= float(h) for l, v, h in zip(o._lo, q, o._hi))
        with pytest.raises(IndexError):
            o.Query(q)
        with pytest.raises(IndexError):
            o.rQuery(np.tile(q, (700, 1)))
        with pytest.raises(IndexError):
            o.rQuery(torch.from_numpy(np.tile(q, (700, 1))).cuda())
    if dim == 3:
        o.trajectories(q[None], np.zeros((1, 3)), 1e-30, 1)
        assert o.lost == 1
