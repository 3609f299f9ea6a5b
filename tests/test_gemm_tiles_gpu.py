"""The tiled weight layout and the skinny GEMM's split of a row tile over the warps of an SM, at the edges of both: one row,
ragged row tiles, columns that end inside a tile (Q8_0), parts of one super-block, parts of unequal length, more row tiles
than warp groups."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _upload(llb, packs, dev, ty, raw, rows, cols):
    w = dev(llb.lib().llb_b200_weight_bytes(packs.FMT[ty], rows, cols))
    llb.check(llb.lib().llb_b200_weight_upload(packs.FMT[ty], rows, cols, raw.ctypes.data, 0, w.ptr), "weight_upload")
    return w


@pytest.mark.parametrize("ty,rows,cols", [("Q8_0", 17, 96), ("Q8_0", 1, 288), ("Q6_K", 31, 512), ("Q5_K", 15, 256)])
def test_tiles_hold_every_weight(llb, packs, dev, ty, rows, cols):
    raw = packs.QUANT[ty](torch.from_numpy(np.random.default_rng(5).standard_normal((rows, cols), dtype=np.float32)))
    out = dev(rows * cols * 4)
    w = _upload(llb, packs, dev, ty, raw.numpy(), rows, cols)
    llb.check(llb.lib().llb_b200_dequant(packs.FMT[ty], rows, cols, w.ptr, 0, rows, out.ptr), "dequant")
    ref = packs.dequant(ty, raw, rows, cols).numpy()
    assert np.array_equal(out.read((rows, cols), np.float32).view(np.uint32), ref.view(np.uint32))


@pytest.fixture
def mma_sync(llb):
    """Q4_K launches stay on the mma.sync kernel, whose tiles, rings and folded form these are."""
    was = llb.lib().llb_b200_use_tcgen05(0)
    yield
    llb.lib().llb_b200_use_tcgen05(was)


@pytest.mark.parametrize("ksplit", [0, 1, 3])
@pytest.mark.parametrize("rows,K,T", [(1, 256, 1), (16, 1024, 1), (17, 3328, 3), (100, 2048, 8), (2500, 1280, 4), (40, 4096, 16), (19200, 2560, 9), (19216, 2560, 16)])
@pytest.mark.parametrize("ty", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_row_tiles_shared_by_warps(llb, packs, dev, mma_sync, ty, rows, K, T, ksplit):
    """(19200 rows of ten super-blocks are the most tiles before Q4_K's scales go into the codes at nine rows and more, 19216 the fewest behind)"""
    rng = np.random.default_rng(rows + K)
    raw = packs.QUANT[ty](torch.from_numpy(rng.standard_normal((rows, K), dtype=np.float32) * 0.05))
    x = rng.standard_normal((T, K), dtype=np.float32)
    w, xd, y = _upload(llb, packs, dev, ty, raw.numpy(), rows, K), dev(x.nbytes).write(x), dev(T * rows * 4)
    L = llb.lib()
    xp = llb.handle(L.llb_b200_xp_new(K, T, 2), "xp_new")
    llb.check(L.llb_b200_xp_set_f32(xp, xd.ptr), "xp_set")
    llb.gemm(packs.FMT[ty], [w.ptr], [rows], [y.ptr], K, xp, ksplit)
    got = y.read((T, rows), np.float32)
    L.llb_b200_xp_free(xp)
    deq = packs.dequant(ty, raw, rows, K).numpy().astype(np.float64)
    # activations to about 22 bits, f32 sums: 1e-5 of the sum of the products' magnitudes
    assert np.all(np.abs(got - x.astype(np.float64) @ deq.T) <= 1e-5 * (np.abs(x).astype(np.float64) @ np.abs(deq).T) + 1e-6)
    assert L.llb_b200_wait_errors() == 0
