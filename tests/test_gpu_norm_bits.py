"""The float64 |B| of the ingest is the correctly rounded root, bit for bit, in
every magnitude range (integer root) and outside it (zeros, subnormals,
infinities, NaN)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows in meshgrid order with x slowest and with x fastest, and in no order: the three fill kernels
@pytest.mark.parametrize("order", ["ij", "xfast", "shuffled"])
@pytest.mark.parametrize("kind", ["unit", "squares", "wide", "edge"])
def test_norm_is_the_rounded_root(kind, order):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from arbinterp_gb300 import tricubic
    rng = np.random.default_rng(11)
    n = (24, 18, 20)
    N = int(np.prod(n))
    B = rng.standard_normal((N, 3))
    if kind == "squares":          # roots that are exact, and the neighbours of such squares
        k = rng.integers(1, 1 << 26, N).astype(np.float64)
        B = np.stack([k, np.zeros(N), np.zeros(N)], 1)
        B[::3, 0] = np.nextafter(k[::3], 0)
        B[1::3, 1] = k[1::3] * 2.0 ** -27
    if kind == "wide":
        B = B * np.exp2(rng.uniform(-480, 480, (N, 1)))
    if kind == "edge":
        B[:400] = rng.choice([0.0, 5e-324, 1e-310, 1e-160, 1e154, 1.5e154, 1e300, np.inf, np.nan], (400, 3))
    G = np.meshgrid(*[np.linspace(0.0, 1.0, m) for m in n], indexing="ij")
    rows = np.stack([g.reshape(-1) for g in G] + [B[:, a] for a in range(3)], 1)
    want = rows.reshape(*n, 6).transpose(2, 1, 0, 3).reshape(N, 6)          # z slowest, x fastest
    if order == "xfast":
        rows = want.copy()
    elif order == "shuffled":
        rows = rows[rng.permutation(N)]
    with np.errstate(all="ignore"):
        w = np.sqrt((want[:, 3] * want[:, 3] + want[:, 4] * want[:, 4]) + want[:, 5] * want[:, 5])
    for mode in ("norm", "both"):
        got = tricubic(rows, "quiet", mode=mode).Bn
        assert np.array_equal(np.isnan(got), np.isnan(w))
        assert np.array_equal(got[~np.isnan(w)].view(np.int64), w[~np.isnan(w)].view(np.int64))
