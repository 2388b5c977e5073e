"""The benchmark's view batches: a batch has a wave schedule of its own, so it evaluates another number of records than its
views alone; what it composites is the same."""
import argparse

import pytest
import torch

import bench
from mlp_splatting_b200 import _lib as L
from mlp_splatting_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def test_a_batch_with_windows_of_its_own_is_sized_and_counted(monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    monkeypatch.setitem(syn.WORKLOADS, "views4", dict(n=30_000, W=256, H=160, mu=-4.6, views=4, seed=5))
    args = argparse.Namespace(width=0, height=0, primitives=0, precision="fp16", encoder="integrated", view_batch=16)
    wl = bench.Workload("views4", args, torch.device("cuda", 0), 1, 0, L.load())
    stats = wl.size_and_count()
    (batch, index), = wl.batches
    alone = wl.r
    assert alone._waves.get(wl.ps.n, 32, wl.prec)[0] != batch._waves.get(wl.ps.n, 32, wl.prec)[0]
    assert index == [0, 1, 2, 3] and stats.used <= stats.records == batch.last_stats.records < batch.lead.max_records
    wl.frame()
    assert batch.last_stats.used == stats.used
    for (cam, _rows), (ro, rd), view in zip(wl.units, wl.dev_rays, batch.views):
        rgb, alpha = alone.render(wl.ps, ro, rd, bench.THRESHOLD, view=cam["view"], proj=cam["proj"], precision=wl.prec,
                                  rays_normalized=True)
        assert torch.equal(rgb, view.rgb) and torch.equal(alpha, view.alpha)
