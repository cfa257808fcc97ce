"""The U-Net convolutions that march over planes, at the sizes where a march can
go wrong: the smallest volume, more planes than a march holds and a last march
that is not full, odd numbers of 8-row tiles, several volumes in a batch. Held
to the same bounds against the mma.sync path as full volumes are
(test_gpu_unet.py): the two share the BF16 rounding points and differ only in
the order of FP32 sums, which a smaller volume makes shorter.
"""
import pytest

from test_gpu_unet import test_tcgen05_matches_mma_sync as matches_mma_sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4, 8, 16), (1, 4, 24, 48), (1, 36, 8, 16), (3, 20, 40, 32),
                                   (2, 68, 16, 16)])
def test_marching_convolutions_match_mma_sync(nusif_lib, shape):
    matches_mma_sync(nusif_lib, shape)
