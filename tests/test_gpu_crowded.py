"""Bins that hold far more queries than the mean are cut into shares: results
do not depend on how the queries are spread over bins and CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _crowd(lo, hi, n, where, seed):
    """n points: all in one cell, all in one bin, most around the middle, or two crowds and a few strays."""
    rng = np.random.default_rng(seed)
    lo, hi = np.array(lo), np.array(hi)
    mid = 0.5 * (lo + hi)
    if where == "cell":
        return mid + 1e-3 * (hi - lo) * rng.random((n, len(lo)))
    if where == "bin":
        return lo + 0.15 * (hi - lo) * rng.random((n, len(lo)))
    if where == "middle":
        return np.clip(mid + 0.1 * (hi - lo) * rng.standard_normal((n, len(lo))), lo, hi - 1e-9 * (hi - lo))
    q = lo + (hi - lo) * (1e-9 + (1 - 2e-9) * rng.random((n, len(lo))))
    q[: n // 2] = lo + 0.1 * (q[: n // 2] - lo)
    q[n // 2: n - n // 50] = hi - 0.1 * (hi - q[n // 2: n - n // 50])
    return q


# share boundaries: one record either side of 512, of a whole number of shares, and many shares
@pytest.mark.parametrize("n", [511, 512, 513, 1025, 20000])
@pytest.mark.parametrize("where", ["cell", "bin", "middle", "two"])
@pytest.mark.parametrize("mode", ["scalar", "vector", "both", "quad"])
def test_crowded_bins_keep_the_results(mode, where, n):
    from arbinterp_gb300 import quadcubic, synth, tricubic
    if mode == "quad":
        f, cls, kw = synth.moving_gaussian_field4((13, 9, 10, 8), seed=2), quadcubic, {}
    elif mode == "scalar":
        f, cls, kw = synth.gaussian_field3((29, 20, 21), seed=2), tricubic, {}
    else:
        f, cls, kw = synth.dipole_field3((29, 20, 21), seed=2), tricubic, {"mode": mode}
    for prec in ("mixed", "fp64"):
        o = cls(f.numpy(), "quiet", precision=prec, strategy="otf", sort_threshold=0, **kw)
        p = cls(f.numpy(), "quiet", precision=prec, strategy="otf", sort_threshold=1 << 40, **kw)
        q = _crowd([float(v) for v in o._lo], [float(v) for v in o._hi], n, where, n)
        got, want = o.Query(q.copy()), p.Query(q.copy())
        assert np.array_equal(o.queryInds, p.queryInds)
        # float64 takes another scale in a staged bin than in a gathered block: there the same rows twice over
        # (other shares, same bins) give the same bits; its accuracy is tested by itself
        twice = o.Query(np.concatenate([q, q]))
        for a, b, c in zip(*(r if isinstance(r, tuple) else (r,) for r in (got, want, twice))):
            if prec == "mixed":
                assert np.array_equal(a, b, equal_nan=True)
            assert np.array_equal(a, c[:n], equal_nan=True) and np.array_equal(a, c[n:], equal_nan=True)


@pytest.mark.parametrize("n", [31, 33, 513, 9000])
@pytest.mark.parametrize("where", ["cell", "middle", "two"])
def test_crowded_adjoint(where, n):
    """The per-warp scatter with up to 32 lanes in one cell, against the float64 adjoint: float32 sums of n terms."""
    import torch
    from arbinterp_gb300 import synth
    from arbinterp_gb300.autograd import TricubicField
    f = synth.gaussian_field3((29, 20, 21), seed=2)
    res = {}
    for prec, binned in (("fp64", False), ("mixed", False), ("mixed", True)):
        F = TricubicField(f.numpy(), precision=prec, binned_adjoint=binned)
        q = _crowd([float(v) for v in F.interp._lo], [float(v) for v in F.interp._hi], n, where, n)
        rng = np.random.default_rng(n)
        v = F.initial_values().requires_grad_(True)
        x = torch.from_numpy(q).cuda().requires_grad_(True)
        up = (torch.from_numpy(rng.standard_normal(n)).cuda(), torch.from_numpy(0.1 * rng.standard_normal((n, 3))).cuda())
        res[prec, binned] = torch.autograd.grad(F(v, x), (v, x), up)
    ref = res["fp64", False]
    # largest |dL/df| of n terms of magnitude <= 60 (upstream 1 + 0.1 * 3 / h), summed in float32 in any order
    lim = 60 * 2.0 ** -24 * (n + 16)
    assert (res["mixed", True][0] - ref[0]).abs().max() <= lim
    assert torch.equal(res["mixed", True][1], res["mixed", False][1])
