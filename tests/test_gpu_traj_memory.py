"""Trajectories on a grid that leaves no room for the packed |B| run without it, with the
same bits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_trajectories_without_room_for_pairs(monkeypatch):
    import torch
    from arbinterp_gb300 import synth, tricubic
    o = tricubic(synth.dipole_field3((20, 18, 17), seed=3), "quiet", mode="both", precision="mixed")
    lo = torch.tensor([float(v) for v in o._lo], dtype=torch.float64, device="cuda")
    hi = torch.tensor([float(v) for v in o._hi], dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    x = lo + (hi - lo) * (0.2 + 0.6 * torch.rand(3000, 3, generator=g, device="cuda", dtype=torch.float64))
    v = 0.05 * (hi - lo) * torch.randn(3000, 3, generator=g, device="cuda", dtype=torch.float64)
    want = o.trajectories(x, v, 0.01, 7, coef=-1e-3)
    empty, refused = torch.empty, []

    def full(*size, **kw):
        if size == (2 * o._npts,):
            refused.append(size)
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", full)
    got = o.trajectories(x, v, 0.01, 7, coef=-1e-3)
    assert refused
    assert all(torch.equal(torch.nan_to_num(a), torch.nan_to_num(b)) for a, b in zip(want, got))
