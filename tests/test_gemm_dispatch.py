"""Which of the two skinny-GEMM kernels a Q4_K launch takes, and in how many K-slices."""
import ctypes as C

import pytest

Q4_K = 3


def kernel(L, nc, rows, K, ksplit=0, sms=148, alone=True):
    """(2 mma.sync or 3 tcgen05, K-slices)"""
    ks = C.c_int(ksplit)
    return L.llb_b200_gemm_kernel(Q4_K, nc, (rows + 15) // 16, K // 256, sms, int(alone), C.byref(ks)), ks.value


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [8, 16, 32])
@pytest.mark.parametrize("rows,K", [(34816, 5120), (5120, 17408), (6144, 5120), (80, 1280)])
def test_the_setting_decides_for_every_launch(llb, nc, rows, K):
    L = llb.lib()
    was = L.llb_b200_use_tcgen05(0)
    try:
        assert was == 2                                     # the default: by size
        assert all(kernel(L, nc, rows, K, alone=a)[0] == 2 for a in (False, True))
        assert L.llb_b200_use_tcgen05(1) == 0
        assert all(kernel(L, nc, rows, K, alone=a)[0] == 3 for a in (False, True))
    finally:
        assert L.llb_b200_use_tcgen05(was) == 1
    assert kernel(L, nc, 34816, 5120)[0] == 3 and kernel(L, nc, 16, 1024)[0] == 2
    assert kernel(L, 8, rows, K, alone=False)[0] == 2       # a pass of up to four rows
