"""The bytes behind the warm-start network's roofline are those its four
kernels move."""


def test_forward_bytes_hold_no_copy_of_x():
    """960x540x64: x read as FP32 by the first layer and again as the residual,
    three hidden activations of 32 channels in BF16 written and read, the FP32
    output written."""
    import bench
    pix = 960 * 540
    want = pix * (64 * 4 + 3 * (32 * 2 + 32 * 2) + 64 * 4 + 64 * 4)
    assert bench.warmnet_forward_bytes(960, 540, 64) == want
    assert round(want / 1e6, 1) == 597.2
