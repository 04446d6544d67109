"""Which operands the split float32 product takes, by their strides (no GPU is needed to ask)."""
import pytest
import torch


@pytest.mark.parametrize("a_stride,w_stride,rows,fits", [(1600, 1600, 8, True), (1608, 1604, 8, True), (0, 1600, 8, False), (16, 1600, 8, False),
                                                         (1600, 0, 8, False), (0, 1600, 1, True), (1601, 1600, 8, False)])
def test_which_strides_the_split_product_takes(a_stride, w_stride, rows, fits):
    from damendaemon_b200 import kernels
    a = torch.zeros(20000).as_strided((rows, 1600), (a_stride, 1))
    w = torch.zeros(20000).as_strided((8, 1600), (w_stride, 1))
    assert kernels.gemm_split_fits(a, w) == fits
