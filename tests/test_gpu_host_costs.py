"""Costs read where they are in host memory: columns and labels at the edges of
the transform's runs, buffers that start anywhere in a line."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,opt", [(np.float32, {}), (np.float32, {"compute_type": 2}), (np.int32, {}),
                                       (np.float32, {"store": 1})])
@pytest.mark.parametrize("offset", [0, 1, 31])
def test_in_place_equals_staged(ginf, dtype, opt, offset):
    import torch
    for L in (2, 9, 16, 20, 33, 48, 56, 75, 90, 100, 110, 128):  # each compiled transform, and one between
        for W, H, levels in ((3, 4, 1), (31, 5, 3), (33, 4, 2), (97, 3, 1), (255, 5, 2), (257, 6, 3), (513, 3, 1)):
            rs = np.random.RandomState(W + L + offset)
            flat = torch.empty(L * H * W + offset, dtype=torch.float32 if dtype == np.float32 else torch.int32,
                               pin_memory=True)
            D = flat[offset:].view(L, H, W)
            D.copy_(torch.from_numpy(rs.randint(0, 4000, (L, H, W)).astype(dtype)))
            V = synth.random_problem(3, 3, L, 1, model=synth.TRUNC_LINEAR, scale=9.0, trunc=60.0).V.astype(dtype)
            V = torch.from_numpy(V).pin_memory()
            got, mg = ginf.decode_hbp(D, V, synth.TRUNC_LINEAR, levels, 2, want_msgs=True, host_access=ginf.HOST_AUTO,
                                      **opt)
            want, mw = ginf.decode_hbp(D, V, synth.TRUNC_LINEAR, levels, 2, want_msgs=True,
                                       host_access=ginf.HOST_COPY, **opt)
            assert np.array_equal(np.asarray(got)[1:-1, 1:-1], np.asarray(want)[1:-1, 1:-1]), (L, W, H)
            assert np.array_equal(np.asarray(mg).view(np.uint8), np.asarray(mw).view(np.uint8)), (L, W, H)
