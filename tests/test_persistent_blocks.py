"""Blocks of a persistent launch: small batches are spread over a warp per
scheduler, kernels with more than 256 bytes of local memory only while every
run has a warp to itself (CPU)."""

import pytest

SMS = 148


@pytest.mark.parametrize("block,per_sm", [(32, 32), (64, 16), (128, 8), (256, 4), (512, 2), (1024, 1)])
def test_blocks_by_runs(block, per_sm):
    from cubie_b200._native import persistent_blocks
    resident, spread = SMS * per_sm, SMS * 128 // block
    warps = spread * (block // 32)
    for runs in (1, 31, 128, 591, 592, 593, 3000, 9000, 18943, 18944, 18945, 40000, 10 ** 6):
        packed = min(-(-runs // block), resident)
        few = min(max(packed, min(spread, runs)), resident)
        for local in (0, 8, 256):
            assert persistent_blocks(resident, SMS, block, runs, local) == few
        for local in (257, 312, 4032):
            assert persistent_blocks(resident, SMS, block, runs, local) == (few if runs <= warps else packed)
    assert persistent_blocks(resident, SMS, block, 0, 0) == 0


def test_bad_shapes_are_refused():
    from cubie_b200._native import NativeError, persistent_blocks
    for args in ((0, SMS, 128, 1, 0), (1, 0, 128, 1, 0), (1, SMS, 100, 1, 0), (1, SMS, 128, -1, 0), (1, SMS, 128, 1, -1)):
        with pytest.raises(NativeError):
            persistent_blocks(*args)
