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


def test_the_number_of_sms_asked_about_decides(pkg):
    """The launch's kernel and K-slices on 148 SMs, without a device: the same as where such a device is in use."""
    L = pkg.llb.lib()
    assert L.llb_b200_gemm_ksplit(Q4_K, 16, 320, 20, 148) == kernel(L, 16, 5120, 5120, alone=False)[1] == 4
    assert L.llb_b200_gemm_ksplit(Q4_K, 16, 256, 16, 148) == 4
    assert kernel(L, 16, 17408, 5120, alone=False)[0] == 3
    # on few SMs a launch has tiles for all of them whatever the kernel; on very many the tcgen05 kernel's 128-row tiles leave most idle
    assert kernel(L, 16, 2048, 2048, sms=16)[0] == 3 and kernel(L, 16, 2048, 2048, sms=2000)[0] == 2


@pytest.mark.gpu
def test_the_device_in_use_decides_nothing_about_others(llb):
    L = llb.lib()
    assert L.llb_b200_sm_count() == 148
    test_the_number_of_sms_asked_about_decides(type("P", (), {"llb": llb}))


@pytest.mark.parametrize("cap", [8, 16])
@pytest.mark.parametrize("nc", [8, 16, 32])
@pytest.mark.parametrize("fmt", [Q4_K, 9, 4, 1])
def test_a_width_fits_where_a_launch_can_be_made(pkg, fmt, nc, cap):
    """Columns up to 512 super-blocks: no narrower matrix is refused than one that is taken, and each kernel's slices are held against its
    own room."""
    L = pkg.llb.lib()
    fits = [bool(L.llb_b200_gemm_fits(fmt, nc, n, cap)) for n in range(1, 513)]
    assert fits == sorted(fits, reverse=True)
    assert fits[:cap * {8: 13, 16: 7, 32: 4}[nc]] == [True] * (cap * {8: 13, 16: 7, 32: 4}[nc])
    if fmt == Q4_K and nc == 16:
        assert L.llb_b200_gemm_fits(fmt, nc, 14, cap) == 1   # 3584 columns: one slice of the tcgen05 kernel, two of the other one


@pytest.mark.gpu
def test_an_engine_keeps_the_kernels_it_was_opened_with(pkg, packs, llb):
    """Six rows a pass of a Q4_K model of three super-blocks' width, opened with the tcgen05 kernel asked for; the setting then changes, and
    the cycle graph is captured again for a sampler: the same bits as without the change."""
    import numpy as np
    L = llb.lib()
    cfg = packs.cfg_tiny(d_model=768, d_ff=1024, quant="q4_k_s")
    pack = packs.build_pack(cfg)
    prompt = packs.synth_prompt(3, 21, cfg.vocab_size)
    out = []
    for later in (1, 0, 2):
        was = L.llb_b200_use_tcgen05(1)
        eng = pkg.llb.SpecEngine(pack, None, k=5, max_ctx=96)
        try:
            L.llb_b200_use_tcgen05(later)
            eng.set_sampler(pkg.llb.SmpParams.make(temp=0.8, top_k=20, seed=9))
            eng.prefill(prompt)
            out.append(eng.generate(24))
            assert L.llb_b200_use_tcgen05(later) == later
        finally:
            L.llb_b200_use_tcgen05(was)
            eng.close()
    for ids, top2 in out[1:]:
        assert np.array_equal(ids, out[0][0]) and np.array_equal(top2, out[0][1])
    assert L.llb_b200_wait_errors() == 0


@pytest.mark.parametrize("nc,rows,K,which", [
    # measured on 148 SMs at the most rows of a width, the other kernel at least 5 % slower at its best
    (8, 40000, 1024, 3), (8, 10240, 5120, 3), (8, 2048, 2048, 2), (8, 17408, 5120, 2), (8, 2285, 8192, 2),
    (16, 34816, 5120, 3), (16, 24576, 4096, 3), (16, 10240, 5120, 3), (16, 2048, 2048, 2), (16, 9216, 2048, 2), (16, 12349, 2816, 2),
    (32, 34816, 5120, 3), (32, 5120, 17408, 3), (32, 5120, 5120, 3), (32, 16384, 2048, 3), (32, 2048, 2048, 2)])
def test_the_operator_takes_the_faster_kernel(pkg, nc, rows, K, which):
    assert kernel(pkg.llb.lib(), nc, rows, K)[0] == which


def test_no_rows_and_no_sms_are_questions_too(pkg):
    L = pkg.llb.lib()
    for nc in (8, 16, 32):
        for alone in (False, True):
            assert kernel(L, nc, 0, 5120, alone=alone)[1] >= 1 and kernel(L, nc, 0, 5120, ksplit=4, alone=alone)[1] == 4
            assert kernel(L, nc, 5120, 5120, sms=0, alone=alone)[1] >= 1
