"""Trajectory inputs that change no result: the order in which threads take the
particles, and |B| as packed (hi, lo) pairs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 1000, (1 << 17) + 5])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("mode", ["scalar", "both"])
def test_order_and_pairs_keep_the_bits(mode, prec, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from arbinterp_gb300 import _lib, synth, tricubic
    L = _lib.lib()
    f = synth.dipole_field3((20, 17, 15), seed=3) if mode == "both" else synth.gaussian_field3((20, 17, 15), seed=3)
    o = tricubic(f.cuda(), "quiet", precision=prec, **({"mode": "both"} if mode == "both" else {}))
    rng = np.random.default_rng(n)
    lo, hi = (np.array([float(v) for v in b]) for b in (o._lo, o._hi))
    x = lo + (hi - lo) * rng.uniform(-0.05, 1.05, (n, 3))
    x[::50] = np.nan
    start = torch.from_numpy(np.concatenate([x, 0.05 * rng.standard_normal((n, 3))], 1)).cuda()
    code = _lib.PREC_MIXED if prec == "mixed" else _lib.PREC_FP64
    if prec == "fp64":
        o._grid64
    keys = torch.empty(n, dtype=torch.int32, device="cuda")
    _lib.check(L.arb_zorder_keys(o._g, start.data_ptr(), n, keys.data_ptr(), None), "keys")
    bad = ~torch.isfinite(start[:, :3]).all(1)
    assert ((keys == 1 << 30) == bad).all() and (keys >= 0).all() and (keys[~bad] < 1 << 30).all()
    pairs = None
    if mode == "both" and prec == "mixed":
        pairs = torch.empty(2 * o._npts, dtype=torch.float32, device="cuda")
        _lib.check(L.arb_norm_pairs(o._g, pairs.data_ptr(), None), "pairs")
    got = []
    for order in (None, torch.argsort(keys), torch.randperm(n, device="cuda")):
        for p in (None, pairs):
            st, path = start.clone(), torch.empty((3, n, 6), dtype=torch.float64, device="cuda")
            lost = torch.zeros(1, dtype=torch.int64, device="cuda")
            _lib.check(L.arb_rk4_trajectories_ordered(
                o._g, code, None if p is None else p.data_ptr(), None if order is None else order.data_ptr(),
                st.data_ptr(), n, 0.02, 6, -1e-2, (ctypes.c_double * 3)(0.0, 0.0, -0.1), path.data_ptr(), 2,
                lost.data_ptr(), None), "rk4")
            torch.cuda.synchronize()
            got.append((st.view(torch.int64), path.view(torch.int64), lost))
    for g in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], g))
