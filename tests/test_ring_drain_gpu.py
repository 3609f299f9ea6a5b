"""A wait of the skinny GEMM's ring that runs out (nothing faults: the stage was simply never requested): the block must not
leave while copies it did request are still on their way into its shared memory."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1, 2000])
def test_a_ring_wait_that_runs_out_leaves_nothing_in_flight(llb, packs, dev, limit):
    L = llb.lib()
    assert L.llb_b200_wait_errors() == 0
    assert L.llb_b200_wait_selftest(2, limit) == 0
    assert L.llb_b200_wait_errors() == 1          # 2: a requested copy had not landed
    assert L.llb_b200_wait_errors_clear() == 0
    rows, K, T, fmt = 33, 1024, 3, packs.FMT["Q4_K"]   # and the device still computes
    raw = packs.QUANT["Q4_K"](torch.from_numpy(np.random.default_rng(1).standard_normal((rows, K), dtype=np.float32)))
    x = np.random.default_rng(2).standard_normal((T, K), dtype=np.float32)
    w, xd, y = dev(L.llb_b200_weight_bytes(fmt, rows, K)), dev(x.nbytes).write(x), dev(T * rows * 4)
    llb.check(L.llb_b200_weight_upload(fmt, rows, K, raw.numpy().ctypes.data, 0, w.ptr), "weight_upload")
    xp = llb.handle(L.llb_b200_xp_new(K, T, 2), "xp_new")
    llb.check(L.llb_b200_xp_set_f32(xp, xd.ptr), "xp_set")
    llb.gemm(fmt, [w.ptr], [rows], [y.ptr], K, xp)
    got = y.read((T, rows), np.float32)
    L.llb_b200_xp_free(xp)
    deq = packs.dequant("Q4_K", raw, rows, K).numpy().astype(np.float64)
    assert np.all(np.abs(got - x.astype(np.float64) @ deq.T) <= 1e-5 * (np.abs(x).astype(np.float64) @ np.abs(deq).T))
    assert L.llb_b200_wait_errors() == 0
