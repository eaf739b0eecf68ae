"""Rows binned once (arb_query_bin) and evaluated on other fields of the same axes
(arb_query_eval_binned): the descriptors may differ in field count and bin shift,
which decide whether a call groups the records by bank class.

Mixed precision: the bits of the row path.  Float64: staged bins and gathered
blocks take different scales, both within 64 units of 2^-53 of the largest sample
(a derivative per cell spacing), so 128 between them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _objects(dim, prec):
    """One interpolant a mode, on the same axes (not multiples of a bin)."""
    from arbinterp_gb300 import quadcubic, synth, tricubic
    if dim == 3:
        s, b = synth.gaussian_field3((30, 21, 23), h=(0.1, 0.1, 0.1), seed=4).numpy(), None
        rng = np.random.default_rng(5)
        cls = tricubic
    else:
        s = synth.moving_gaussian_field4((13, 9, 10, 8), seed=4).numpy()
        rng = np.random.default_rng(6)
        cls = quadcubic
    comps = np.stack([np.cos(k + s[:, dim] * 3) + 0.1 * rng.standard_normal(len(s)) for k in range(3)], 1)
    b = np.concatenate([s[:, :dim], comps], 1)
    kw = dict(precision=prec, strategy="otf")
    return {1: cls(s, "quiet", **kw), 3: cls(b, "quiet", mode="vector", **kw), 4: cls(b, "quiet", mode="both", **kw)}


# rows a bin: below every line, between the lines of three fields and of others (64, 128), and dense
@pytest.mark.parametrize("rows", [30, 90, 150])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("dim", [3, 4])
def test_bins_serve_every_field_count_and_shift(dim, prec, rows):
    import torch
    from arbinterp_gb300 import _lib
    L = _lib.lib()
    objs = _objects(dim, prec)
    o = objs[1]
    lo = np.array([float(v) for v in o._lo])
    hi = np.array([float(v) for v in o._hi])
    edge = 8 if dim == 3 else 4
    n = rows * int(np.prod([(m - 3 + edge - 1) // edge for m in o._n]))
    rng = np.random.default_rng(rows)
    q = lo + (hi - lo) * (1e-9 + (1 - 2e-9) * rng.random((n, dim)))
    q[::37, 0] = lo[0] - 1.0                     # outside
    q[5::41, 1] = np.nan
    qd = torch.from_numpy(q).cuda()
    pc = _lib.PREC_FP64 if prec == "fp64" else _lib.PREC_MIXED
    s = torch.cuda.current_stream().cuda_stream
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    shifts = (2, 3, 4) if dim == 3 else (1, 2, 3)
    want, scale = {}, {}
    for F, p in objs.items():
        p.sort_threshold = 1 << 40
        r = p.Query(q.copy())
        want[F] = [r] if F == 3 else list(r)
        scale[F] = float(p._grid64.abs().max())
    h = np.array([float(v) for v in o._h])

    def descr(F, shift):
        g = _lib.ArbGrid()
        ctypes.memmove(ctypes.byref(g), ctypes.byref(objs[F]._g), ctypes.sizeof(g))
        g.bin_shift = shift
        return g
    need = max(int(L.arb_query_sorted_work_bytes(descr(F, k), pc, n)) for F in objs for k in shifts)
    for Fb, kb in [(F, shifts[1]) for F in objs] + [(1, shifts[0]), (3, shifts[2])]:
        ws = torch.full((need,), 0xA5, dtype=torch.uint8, device="cuda")
        none = _lib.ArbQueryOut()
        assert L.arb_query_bin(descr(Fb, kb), pc, qd.data_ptr(), n, dim, 0, none, ws.data_ptr(), need, st.data_ptr(), s) == 0
        for Fe in objs:
            for ke in shifts:
                R = {1: 4 if dim == 3 else 8, 3: 4, 4: 8}[Fe]
                out = torch.full((n, R), -7.0, dtype=torch.float64, device="cuda")
                at = lambda c: out.data_ptr() + 8 * c  # noqa: E731
                ao = _lib.ArbQueryOut(at(0) if Fe >= 3 else None, None if Fe == 3 else at(0 if Fe == 1 else 3),
                                      None if Fe == 3 else at(1 if Fe == 1 else 4), None, None, None, R, R, R)
                assert L.arb_query_eval_binned(descr(Fe, ke), pc, 0, n, ao, ws.data_ptr(), need, s) == 0
                r = out.cpu().numpy()
                cols = {1: [r[:, :1], r[:, 1:1 + dim]], 3: [r[:, :3]], 4: [r[:, :3], r[:, 3:4], r[:, 4:4 + dim]]}[Fe]
                for i, (got, ref) in enumerate(zip(cols, want[Fe])):
                    if prec == "mixed":
                        assert np.array_equal(got, ref, equal_nan=True), (Fb, kb, Fe, ke)
                        continue
                    grad = Fe != 3 and i == len(cols) - 1
                    assert np.array_equal(np.isnan(got), np.isnan(ref))
                    err = np.nan_to_num(np.abs(got - ref) * (h if grad else 1.0))
                    assert err.max() <= 128 * 2.0 ** -53 * scale[Fe], (Fb, kb, Fe, ke)
    assert int(st.item()) == 0
