"""Weight uploads from device memory as callers have them: odd addresses, a matrix laid out in place, and columns that are not
whole blocks of the format (of which the whole blocks count)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
FMTS = ("Q4_K", "Q5_K", "Q6_K", "Q8_0")


def _raw(packs, ty, rows, cols):
    w = torch.from_numpy(np.random.default_rng(rows + cols).standard_normal((rows, cols), dtype=np.float32))
    return packs.QUANT[ty](w).contiguous()


def _deq(llb, packs, dev, ty, rows, cols, w):
    out = dev(rows * cols * 4)
    llb.check(llb.lib().llb_b200_dequant(packs.FMT[ty], rows, cols, w, 0, rows, out.ptr), "dequant")
    return out.read((rows, cols), np.float32).view(np.uint32)


@pytest.mark.parametrize("off_src,off_dst", [(1, 0), (3, 0), (0, 1), (1, 1), (2, 0)])
@pytest.mark.parametrize("ty", FMTS)
def test_any_address(llb, packs, dev, ty, off_src, off_dst):
    rows, cols, L = 19, 512, llb.lib()
    raw = _raw(packs, ty, rows, cols)
    nb = L.llb_b200_weight_bytes(packs.FMT[ty], rows, cols)
    src, dst = dev(raw.numel() + 16), dev(nb + 16)
    src.write(np.concatenate([np.zeros(off_src, np.uint8), raw.numpy().reshape(-1)]))
    llb.check(L.llb_b200_weight_upload(packs.FMT[ty], rows, cols, src.ptr + off_src, 1, dst.ptr + off_dst), "weight_upload")
    ref = packs.dequant(ty, raw, rows, cols).numpy().view(np.uint32)
    assert np.array_equal(_deq(llb, packs, dev, ty, rows, cols, dst.ptr + off_dst), ref)


@pytest.mark.parametrize("shift", [0, 64])
@pytest.mark.parametrize("ty", FMTS)
def test_in_place(llb, packs, dev, ty, shift):
    rows, cols, L = 80, 1024, llb.lib()
    raw = _raw(packs, ty, rows, cols)
    buf = dev(L.llb_b200_weight_bytes(packs.FMT[ty], rows, cols) + raw.numel() + 64)
    buf.write(np.concatenate([np.zeros(shift, np.uint8), raw.numpy().reshape(-1)]))
    llb.check(L.llb_b200_weight_upload(packs.FMT[ty], rows, cols, buf.ptr + shift, 1, buf.ptr), "weight_upload")
    assert np.array_equal(_deq(llb, packs, dev, ty, rows, cols, buf.ptr), packs.dequant(ty, raw, rows, cols).numpy().view(np.uint32))


@pytest.mark.parametrize("on_device", [0, 1])
@pytest.mark.parametrize("ty,cols,whole", [("Q4_K", 300, 256), ("Q5_K", 700, 512), ("Q6_K", 500, 256)])
def test_columns_past_the_last_whole_block(llb, packs, dev, ty, cols, whole, on_device):
    rows, L = 17, llb.lib()
    raw = _raw(packs, ty, rows, whole)           # a row's bytes are those of its whole blocks
    w = dev(L.llb_b200_weight_bytes(packs.FMT[ty], rows, cols))
    src = dev(raw.numel()).write(raw.numpy()) if on_device else None
    llb.check(L.llb_b200_weight_upload(packs.FMT[ty], rows, cols, src.ptr if on_device else raw.numpy().ctypes.data, on_device, w.ptr), "weight_upload")
    got = _deq(llb, packs, dev, ty, rows, cols, w.ptr)
    assert np.array_equal(got[:, :whole], packs.dequant(ty, raw, rows, whole).numpy().view(np.uint32))
    assert not np.any(got[:, whole:] & 0x7fffffff)


@pytest.mark.parametrize("ty", FMTS)
def test_a_gemm_behind_an_upload_sees_it(llb, packs, dev, ty):
    """Uploads and GEMMs in turn with no synchronisation between them: a GEMM's first weight copies start before the kernels
    in front of it are done, but not before the upload is."""
    rows, cols, T, n, L, fmt = 4096, 2048, 4, 12, llb.lib(), packs.FMT[ty]
    rng = np.random.default_rng(8)
    base = _raw(packs, ty, rows, cols)
    srcs = [base, torch.flip(base, [0]).contiguous()]        # the same rows the other way round
    x = rng.standard_normal((T, cols), dtype=np.float32)
    w, xd = dev(L.llb_b200_weight_bytes(fmt, rows, cols)), dev(x.nbytes).write(x)
    dsrc, outs = [dev(s.numel()).write(s.numpy()) for s in srcs], [dev(T * rows * 4) for _ in range(n)]
    xp = llb.handle(L.llb_b200_xp_new(cols, T, 2), "xp_new")
    llb.check(L.llb_b200_xp_set_f32(xp, xd.ptr), "xp_set")
    for i in range(n):
        llb.check(L.llb_b200_weight_upload(fmt, rows, cols, dsrc[i & 1].ptr, 1, w.ptr), "weight_upload")
        llb.gemm(fmt, [w.ptr], [rows], [outs[i].ptr], cols, xp)
    got = [o.read((T, rows), np.float32) for o in outs]
    L.llb_b200_xp_free(xp)
    for i in range(n):
        assert np.array_equal(got[i], got[i & 1])
    assert np.array_equal(got[0], got[1][:, ::-1])


@pytest.mark.parametrize("ty,cols", [("Q6_K", 4096), ("Q4_K", 32 * 256)])
def test_host_uploads_larger_than_the_staging_buffer(llb, packs, dev, ty, cols):
    """More than 32 MB go through the buffer in whole row tiles; the last piece ends inside one."""
    L, rows = llb.lib(), (70 << 20) // packs.row_bytes(ty, cols) | 1
    raw = _raw(packs, ty, 33, cols).repeat(-(-rows // 33), 1)[:rows].contiguous()
    w = dev(L.llb_b200_weight_bytes(packs.FMT[ty], rows, cols))
    llb.check(L.llb_b200_weight_upload(packs.FMT[ty], rows, cols, raw.numpy().ctypes.data, 0, w.ptr), "weight_upload")
    ids = np.array(sorted({0, 1, 15, 16, rows // 3, rows // 2, rows - 17, rows - 1} | set(range(0, rows, 97))), np.int32)
    d, out = dev(ids.nbytes).write(ids), dev(len(ids) * cols * 4)
    llb.check(L.llb_b200_dequant(packs.FMT[ty], rows, cols, w.ptr, d.ptr, len(ids), out.ptr), "dequant")
    ref = packs.dequant(ty, raw[torch.from_numpy(ids).long()].contiguous(), len(ids), cols).numpy()
    assert np.array_equal(out.read((len(ids), cols), np.float32).view(np.uint32), ref.view(np.uint32))
