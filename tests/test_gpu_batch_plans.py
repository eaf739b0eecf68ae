"""Plans of a batch belong to the kernels they were measured on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_batch_plans_of_other_kernels_are_measured_again(tmp_path, monkeypatch):
    import torch
    from arbinterp_gb300 import autotune, synth
    from arbinterp_gb300.batched import TILE_CHOICES, BatchedTricubic
    monkeypatch.setenv("ARBINTERP_TUNE_DIR", str(tmp_path))
    monkeypatch.setattr(autotune, "_MEM", {})
    fields = [synth.gaussian_field3((9, 9, 9), h=(0.1, 0.1, 0.1), seed=s) for s in (1, 2)]
    lo = np.array([float(v) for v in BatchedTricubic(fields[:1]).interps[0]._lo])
    q = torch.from_numpy(np.tile(lo + 0.05, (200, 1))).cuda()

    def plan():
        b = BatchedTricubic(fields, precision="fp64")
        b.query(q, [100, 100])
        return b.tile_rows
    assert plan() in TILE_CHOICES
    for key in list(autotune._MEM):
        autotune._MEM[key] = {"tile_rows": 3, "table_ratio": None, "ms": 0.0}
        autotune._store(key, autotune._MEM[key])
    assert plan() == 3                             # kept for these kernels, in memory
    autotune._MEM.clear()
    assert plan() == 3                             # and in the file
    monkeypatch.setattr(autotune, "KERNELS", autotune.KERNELS + 1)
    autotune._MEM.clear()
    assert plan() in TILE_CHOICES
