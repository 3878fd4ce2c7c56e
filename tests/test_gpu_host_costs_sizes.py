"""Costs read in place from host memory on either side of the node count from
which on the wide transform reads them, at the edges of its runs."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,opt", [(np.float32, {}), (np.float32, {"compute_type": 2}), (np.int32, {}),
                                       (np.float32, {"store": 1})])
@pytest.mark.parametrize("offset", [0, 1, 31])
def test_in_place_equals_staged(ginf, dtype, opt, offset):
    import torch
    for L in (2, 9, 20, 48, 90, 128):
        for W, H, levels in ((181, 181, 2), (182, 181, 2), (97, 339, 1), (255, 129, 3), (257, 129, 1), (513, 65, 2),
                             (33, 995, 2)):
            rs = np.random.RandomState(W + L + offset)
            flat = torch.empty(L * H * W + offset, dtype=torch.float32 if dtype == np.float32 else torch.int32,
                               pin_memory=True)
            D = flat[offset:].view(L, H, W)
            D.copy_(torch.from_numpy(rs.randint(0, 4000, (L, H, W)).astype(dtype)))
            V = synth.random_problem(3, 3, L, 1, model=synth.TRUNC_LINEAR, scale=9.0, trunc=60.0).V.astype(dtype)
            V = torch.from_numpy(V).pin_memory()
            got, want = (ginf.decode_hbp(D, V, synth.TRUNC_LINEAR, levels, 3, host_access=access, **opt)
                         for access in (ginf.HOST_AUTO, ginf.HOST_COPY))
            assert np.array_equal(np.asarray(got)[1:-1, 1:-1], np.asarray(want)[1:-1, 1:-1]), (L, W, H)
