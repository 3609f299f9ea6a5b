"""Kernels fetched by name leave weights in the layout that the other entry points read."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [1, 5, 100])
@pytest.mark.parametrize("ty", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_tiles_by_name(llb, packs, dev, ty, grid):
    L, rows, cols, fmt = llb.lib(), 37, 768, packs.FMT[ty]
    k = L.llb_b200_kernel_by_name(b"llb_b200_k_to_tiles")
    assert k
    assert not L.llb_b200_kernel_by_name(b"llb_b200_k_repack_q6k")    # its 224-byte blocks are no layout of this library
    raw = packs.QUANT[ty](torch.from_numpy(np.random.default_rng(6).standard_normal((rows, cols), dtype=np.float32))).contiguous()
    src, w, out = dev(raw.numel()).write(raw.numpy()), dev(L.llb_b200_weight_bytes(fmt, rows, cols)), dev(rows * cols * 4)
    vals = [C.c_int(fmt), C.c_uint64(src.ptr), C.c_int(rows), C.c_int(cols), C.c_uint64(w.ptr)]
    argv = (C.c_void_p * len(vals))(*[C.addressof(v) for v in vals])
    assert L.llb_b200_launch(k, grid, 1, 256, 0, argv, len(vals)) == 0
    llb.check(L.llb_b200_dequant(fmt, rows, cols, w.ptr, 0, rows, out.ptr), "dequant")
    ref = packs.dequant(ty, raw, rows, cols).numpy()
    assert np.array_equal(out.read((rows, cols), np.float32).view(np.uint32), ref.view(np.uint32))
