"""The whole table of coefficients where its tiles can go wrong: one tile, fewer
tiles than groups of warps, rows of cells that end just before, at and after a
tile (32, 42 and 128 cells for four, three and one field), against the float64
solve.

Tolerance: a coefficient is a sum of samples with weights of at most 6^3 in
absolute value together, so half an ulp of its float32 value is at most 2^-17 of
the largest sample and the three-part FP16 split (2^-33 a sample) far below that;
2^-16 covers both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("mode,nx", [("both", 4), ("both", 32), ("both", 36), ("both", 40), ("vector", 44), ("vector", 45),
                                     ("vector", 46), ("vector", 90), ("norm", 130), ("norm", 132), ("norm", 134)])
@pytest.mark.parametrize("ny,nz", [(4, 4), (5, 4), (24, 17)])
def test_tiles_of_a_full_solve(mode, nx, ny, nz):
    from arbinterp_gb300 import tricubic
    rng = np.random.default_rng(nx + ny)
    ax = [np.arange(n) * 0.5 for n in (nx, ny, nz)]
    pts = np.stack([m.T.reshape(-1) for m in np.meshgrid(*ax, indexing="ij")], 1)
    field = np.concatenate([pts, rng.standard_normal((len(pts), 3))], 1)
    tabs = []
    for precision in ("mixed", "fp64"):
        ip = tricubic(field, "quiet", mode=mode, precision=precision)
        ip.allCoeffs()
        tabs.append(ip._table.cpu().numpy().astype(np.float64))
    assert tabs[0].shape == tabs[1].shape
    np.testing.assert_allclose(tabs[0], tabs[1], rtol=0, atol=2.0 ** -16 * np.abs(field[:, 3:]).max())
