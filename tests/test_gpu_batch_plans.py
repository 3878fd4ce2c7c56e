"""Batch plans: what the autotuner's cache holds, the tile size reported, and
label buckets with several half-sweeps per launch."""
import json

import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


def _problems(labels, W=37, H=23):
    import torch
    out = []
    for L in labels:
        P = synth.random_problem(W, H, L, 40 + L, trunc=2.5)
        out.append((torch.from_numpy(P.D).cuda(), torch.from_numpy(P.V).cuda(), P.model))
    return out, [torch.zeros((H, W), dtype=torch.int32, device="cuda") for _ in out]


@pytest.mark.parametrize("spl", [3, 0])
def test_label_buckets_across_the_grid_barrier(ginf, spl):
    """Several half-sweeps per launch (7 leave a short last launch), every
    bucket's edge label counts, each tile size."""
    problems, labels = _problems((2, 8, 9, 16, 17, 25, 32, 33, 40, 41, 49, 56, 57, 63, 64))
    want = [ginf.decode_hbp(D, V, m, 1, 7).cpu().numpy() for D, V, m in problems]
    for tile in (8, 16, 32):
        for lab in labels:
            lab.zero_()
        with ginf.Batch(problems, labels, 7, tile_nodes=tile, sweeps_per_launch=spl) as b:
            b.run()
            for lab, w in zip(labels, want):
                assert np.array_equal(lab.cpu().numpy(), w), tile
            b.run()  # a replay
            for lab, w in zip(labels, want):
                assert np.array_equal(lab.cpu().numpy(), w), tile


def test_choices_of_other_kernels_are_measured_anew(ginf, tmp_path, monkeypatch):
    """A cache entry whose key names only the mix of grids, as written before
    the key named the device and the kernels, does not decide a plan, stays in
    the file, and the new choice is used from then on."""
    path = tmp_path / "tune.json"
    old = "L16:s9x1,L40:s9x1,it6"
    path.write_text('{\n  "%s": {"tile_nodes": 32, "sweeps_per_launch": 5, "ms": 0.1}\n}\n' % old)
    monkeypatch.setenv("GINF_AUTOTUNE_CACHE", str(path))
    problems, labels = _problems((16, 40))
    with ginf.Batch(problems, labels, 6) as b:
        first = b.config()
    assert first["tuned_now"] is True
    entries = json.loads(path.read_text())
    assert entries[old]["sweeps_per_launch"] == 5 and len(entries) == 2
    with ginf.Batch(problems, labels, 6) as b:
        second = b.config()
    assert second["tuned_now"] is False and second["tile_nodes"] == first["tile_nodes"]


def test_tile_size_reported_is_the_one_in_use(ginf, tmp_path, monkeypatch):
    """Up to 32 labels a tile is a warp's eight nodes, whatever the options
    say; a plan with other grids reports theirs."""
    monkeypatch.setenv("GINF_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    problems, labels = _problems((5, 16, 32))
    for opt in ({"tile_nodes": 32, "sweeps_per_launch": 1}, {"autotune": -1}, {"autotune": 1}, {}):
        with ginf.Batch(problems, labels, 6, **opt) as b:
            assert b.config()["tile_nodes"] == 8, opt
    problems, labels = _problems((16, 40))
    for tile in (8, 16, 32):
        with ginf.Batch(problems, labels, 6, tile_nodes=tile, sweeps_per_launch=1) as b:
            assert b.config()["tile_nodes"] == tile


@pytest.mark.parametrize("spl", [3, 0])
@pytest.mark.parametrize("W,H", [(37, 23), (330, 260)])
def test_groups_of_a_cooperative_launch(ginf, spl, W, H):
    """Label counts between 32 and 64 in one kernel (the small grids) and apart
    (the large ones), beside those that always stay apart."""
    problems, labels = _problems((5, 20, 33, 40, 41, 50, 63, 64), W, H)
    want = [ginf.decode_hbp(D, V, m, 1, 8).cpu().numpy() for D, V, m in problems]
    with ginf.Batch(problems, labels, 8, tile_nodes=16, sweeps_per_launch=spl) as b:
        for _ in range(2):
            b.run()
            for (D, _, _), lab, w in zip(problems, labels, want):
                assert np.array_equal(lab.cpu().numpy(), w), D.shape
                lab.zero_()


def test_time_of_mixed_label_counts_in_cooperative_launches(ginf):
    """Small grids of four label buckets take at most twice the time of as many
    grids of one (about the same; with launches for each bucket three times)."""
    import torch
    times = []
    for counts in ((48, 48, 48, 48, 48), (34, 44, 53, 59, 62)):
        problems, labels = _problems(counts, 60, 50)
        with ginf.Batch(problems, labels, 15, tile_nodes=16, sweeps_per_launch=0) as b:
            best = float("inf")
            for _ in range(6):
                a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                torch.cuda.synchronize()
                a.record()
                b.run()
                e.record()
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(e))
        times.append(best)
    assert times[1] < 2 * times[0], times
